"""GPU drop-in for the reference's contraction backend.

``ContractionBackend.__call__(subscripts, *operands)`` keeps the einsum-string interface of
``pycc/device.py:64-87`` (the ``self.contract`` every CCSD builder calls), but executes each
pairwise contraction in the CUDA library, as one launch of an FP64 strided kernel or, where that
is the shorter, as exact integer products modulo sixteen moduli on the tensor cores
(``csrc/contract_rns.cu``): operand and output permutations become element strides, nothing is
copied in FP64 and nothing crosses PCIe/C2C (the reference copies CPU-resident integrals per call,
``pycc/device.py:71-74``).

Two keyword-only extensions make the builders allocation-free: ``out=`` accumulates into an
existing tensor and ``alpha``/``beta`` give ``out = beta*out + alpha*contract(...)``.
"""
from __future__ import annotations

import ctypes as C
import functools
import itertools
import math

import torch

from . import _lib

MAX_SUB = 4


def _merge(groups):
    """Merge consecutive sub-indices that are contiguous in both tensors (outer -> inner)."""
    groups = [g for g in groups if g[0] != 1]
    out = []
    for e, s0, s1 in groups:
        if out:
            pe, p0, p1 = out[-1]
            if p0 == e * s0 and p1 == e * s1:
                out[-1] = (pe * e, s0, s1)
                continue
        out.append((e, s0, s1))
    return out


def _parse(subscripts):
    s = subscripts.replace(" ", "")
    if "->" not in s:
        raise ValueError("contract: explicit output ('->') required, got %r" % subscripts)
    lhs, rhs = s.split("->")
    ins = lhs.split(",")
    return ins, rhs


class ContractPlan:
    """Sub-index groups of one pairwise contraction for given operand strides."""

    def __init__(self, subscripts, a, b, out_shape=None):
        ins, rhs = _parse(subscripts)
        if len(ins) != 2:
            raise ValueError("contract: exactly two operands supported, got %d" % len(ins))
        sa, sb = ins
        for sub, t in ((sa, a), (sb, b)):
            if len(sub) != t.dim():
                raise ValueError("contract: %r does not match operand of rank %d" % (sub, t.dim()))
            if len(set(sub)) != len(sub):
                raise ValueError("contract: repeated index within an operand (%r)" % sub)
        if len(set(rhs)) != len(rhs):
            raise ValueError("contract: repeated output index (%r)" % rhs)
        ext = {}
        for sub, t in ((sa, a), (sb, b)):
            for c, n in zip(sub, t.shape):
                if ext.setdefault(c, n) != n:
                    raise ValueError("contract: index %r has extents %d and %d" % (c, ext[c], n))
        for c in rhs:
            if c not in ext:
                raise ValueError("contract: output index %r absent from the operands" % c)
        for c in set(sa) | set(sb):
            if c not in rhs and not (c in sa and c in sb):
                raise ValueError("contract: index %r summed over a single operand" % c)
        self.sa, self.sb, self.rhs = sa, sb, rhs
        self.shape = tuple(ext[c] for c in rhs)
        self.ext = ext

    def groups(self, a, b, out):
        sa, sb, rhs, ext = self.sa, self.sb, self.rhs, self.ext
        ast = dict(zip(sa, a.stride()))
        bst = dict(zip(sb, b.stride()))
        cst = dict(zip(rhs, out.stride()))
        M, N, batch = [], [], []
        for c in rhs:
            ia, ib = c in ast, c in bst
            if ia and ib:
                batch.append(c)
            elif ia:
                M.append((ext[c], ast[c], cst[c]))
            else:
                N.append((ext[c], bst[c], cst[c]))
        K = [(ext[c], ast[c], bst[c]) for c in sa if c in bst and c not in cst]
        K.sort(key=lambda g: (-g[1], -g[2]))
        M, N, K = _merge(M), _merge(N), _merge(K)
        if max(len(M), len(N), len(K)) > MAX_SUB:
            raise ValueError("contract: more than %d sub-indices after merging" % MAX_SUB)
        return M, N, K, batch, ast, bst, cst


def _check(t, name):
    if not isinstance(t, torch.Tensor):
        raise TypeError("contract: %s must be a torch.Tensor" % name)
    if not t.is_cuda:
        raise ValueError("contract: %s must be resident on the GPU (no host copies)" % name)
    if t.dtype != torch.float64:
        raise TypeError("contract: %s must be float64, got %s" % (name, t.dtype))


class _Call:
    """The launch arguments of one contraction that its labels, extents and strides fix: the
    sub-index groups as C arrays, the extents and strides of its batch indices, the output shape and
    whether it goes to the residue path."""

    def __init__(self, subscripts, a, b, out):
        plan = ContractPlan(subscripts, a, b)
        self.shape = plan.shape
        if out is None:
            out = torch.empty(plan.shape, dtype=torch.float64, device="meta")
        elif tuple(out.shape) != plan.shape:
            raise ValueError("contract: out has shape %s, expected %s"
                             % (tuple(out.shape), plan.shape))
        M, N, K, batch, ast, bst, cst = plan.groups(a, b, out)
        self.groups = _group_args(M, N, K)
        self.mnk = tuple(math.prod([g[0] for g in G]) for G in (M, N, K))
        self.rns = _takes_rns(*self.mnk)
        # batch indices (present in both operands and the output): one launch per value
        self.batch = [plan.ext[c] for c in batch]
        self.steps = [[8 * st[c] for c in batch] for st in (ast, bst, cst)]

    def offsets(self):
        """Byte offsets of the operands and the output at every value of the batch indices."""
        if not self.batch:
            return ((0, 0, 0),)
        return (tuple([sum(v * s for v, s in zip(vals, step)) for step in self.steps])
                for vals in itertools.product(*[range(n) for n in self.batch]))


_CALLS = {}


def contract_f64(subscripts, a, b, out=None, alpha=1.0, beta=0.0, stream=None):
    """``out = beta*out + alpha * einsum(subscripts, a, b)`` in FP64: on the FP64 kernels, or,
    where that is the shorter (``_takes_rns``), on the tensor cores in residue arithmetic.  Both
    keep every output's error within about K 2^-53 sum |a||b| over its K products (an output for
    which the residues' common scale of a row is too coarse is summed in FP64)."""
    _check(a, "operand 0")
    _check(b, "operand 1")
    if out is not None:
        _check(out, "out")
    key = (subscripts, a.shape, a.stride(), b.shape, b.stride(),
           None if out is None else (out.shape, out.stride()))
    call = _CALLS.get(key)
    if call is None:
        call = _lib.remember(_CALLS, key, _Call(subscripts, a, b, out))
    if out is None:
        out = torch.empty(call.shape, dtype=torch.float64, device=a.device)
        beta = 0.0
    work = _rns_scratch(*call.mnk, out.device, stream) if call.rns else None
    st = _lib.stream_handle(stream)
    pa, pb, pc = a.data_ptr(), b.data_ptr(), out.data_ptr()
    for oa, ob, oc in call.offsets():
        _launch_groups(call.groups, alpha, pa + oa, pb + ob, beta, pc + oc, st, work)
    return out


def _group_args(M, N, K):
    """The three sub-index groups as the library takes them."""
    i64 = _lib.i64s
    out = ()
    for G in (M, N, K):
        out += (len(G), i64([g[0] for g in G]), i64([g[1] for g in G]), i64([g[2] for g in G]))
    return out


def _launch_groups(groups, alpha, pa, pb, beta, pc, st, work=None):
    if work is None:
        _lib.call("pcg_contract_f64", *groups, float(alpha), pa, pb, float(beta), pc, st)
    else:
        _lib.call("pcg_contract_rns_f64", *groups, float(alpha), pa, pb, float(beta), pc,
                  work.data_ptr(), work.numel(), st)


def _launch(M, N, K, alpha, pa, pb, beta, pc, st, work=None):
    _launch_groups(_group_args(M, N, K), alpha, pa, pb, beta, pc, st, work)


# Bytes of scratch of one contraction in residue arithmetic.  8.5 GiB hold 12000 x 12000 x 12000
# (no = 40, nv = 300) in two panels of rows: 38.6 ms, in four panels (8 GiB) 44.2.
RNS_WORK_LIMIT = 17 << 29


@functools.lru_cache(maxsize=4096)
def _rns_work(m, n, k, limit=RNS_WORK_LIMIT):
    """Scratch bytes of an m x n x k contraction in residue arithmetic (0: does not fit)."""
    out = C.c_longlong(0)
    _lib.call("pcg_contract_rns_f64_work", m, n, k, limit, C.byref(out))
    return out.value


@functools.lru_cache(maxsize=4096)
def _takes_rns(m, n, k):
    """Whether an m x n x k contraction runs on the tensor cores in residue arithmetic rather
    than on the FP64 pipe: where its estimated time is the shorter one.

    FP64 pipe: 6 us and 1.05 TFLOP/s.  Residues: 42 us of launches, 50 bytes moved per operand
    element at 5 TB/s, 0.3 ns per step of K (a row's norm), 17 BF16 products over whole 128 x 16 x
    64 tiles at 1.1 PFLOP/s and at least 2.5 us for 128 x 256 of them on an SM, and 13 ps per
    output to rebuild it.  Measured (us, FP64 pipe / residues), where the rule takes the FP64 pipe:
    53 x 53 x 4293 42 / 47, 110 x 21560 x 14 92 / 102, 11 x 75779 x 83 146 / 221, 20 x 20 x 648000
    556 / 713, and on the wrong side by up to 1.4 2809 x 81 x 81 52 / 44, 128 x 128 x 1024 58 / 41;
    where it takes the residues: 60 x 60 x 8640 76 / 56, 14 x 169400 x 110 486 / 458, 180 x 72000 x
    20 518 / 393, 477 x 477 x 477 206 / 44."""
    if min(m, n) < 2 or m * n * k < 1 << 22:
        return False
    up = lambda x, t: -(-x // t) * t
    fp64 = 6e-6 + 2.0 * m * n * k / 1.05e12
    lo, hi = (m, n) if m < n else (n, m)
    gemm = max(34.0 * up(lo, 128) * hi * up(k, 64) / 1.1e15,
               17 * up(lo, 128) // 128 * up(hi, 256) // 256 * 2.5e-6 / 152)
    rns = 42e-6 + 50.0 * (m + n) * k / 5e12 + 0.3e-9 * k + gemm + 13e-12 * m * n
    return rns < fp64


def _rns_scratch(m, n, k, device, stream):
    """Scratch for the call on ``device``, owned by the launching stream, or None when the
    device has no room even for small panels (the FP64 kernel needs none) or is not a GPU."""
    if device.type != "cuda":
        return None
    limit = RNS_WORK_LIMIT
    while limit >= 256 << 20:
        nbytes = _rns_work(m, n, k, limit)
        if not nbytes:
            return None
        try:
            if stream is None:
                return torch.empty(nbytes, dtype=torch.uint8, device=device)
            with torch.cuda.stream(stream):
                return torch.empty(nbytes, dtype=torch.uint8, device=device)
        except torch.cuda.OutOfMemoryError:
            limit = min(limit, nbytes) // 4
    return None


class ContractionBackend:
    """``self.contract`` of the GPU CCSD engine (mirrors ``pycc/device.py:38-87``)."""

    def __init__(self, device1=None, stream=None):
        self.device = "GPU"
        self.device1 = device1 if device1 is not None else torch.device("cuda:0")
        self.stream = stream

    def __call__(self, subscripts, *operands, out=None, alpha=1.0, beta=0.0):
        if len(operands) != 2:
            raise ValueError("contract: the GPU engine contracts operand pairs (got %d)" % len(operands))
        return contract_f64(subscripts, operands[0], operands[1], out=out, alpha=alpha,
                            beta=beta, stream=self.stream)
