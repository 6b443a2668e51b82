"""The three BF16 pieces of an FP64 operand (split-BF16x6), bit by bit against rounding in numpy."""
import numpy as np
import pytest
import torch

from pycc_gb300.tc import FMT_BF16X6, Operand, pack

pytestmark = pytest.mark.gpu


def bf16(x):
    """Nearest BF16 values of float64 ones, ties to even (BF16's normal range)."""
    m, e = np.frexp(x)
    return np.ldexp(np.rint(m * 256.0), e - 8)


def values(n, rng):
    """All magnitudes of the range, ties, values of few bits, zeros of both signs."""
    x = rng.standard_normal(n) * 10.0 ** rng.uniform(-25, 29, n)
    m, e = np.frexp(x)
    few = np.ldexp(np.rint(m * 2.0 ** rng.integers(7, 30, n)), 0)
    x[::3] = np.ldexp(few, rng.integers(-60, 60, n))[::3]
    x[5::17], x[6::19] = 0.0, -0.0
    return x


@pytest.mark.parametrize("rows,k", [(1, 1), (63, 65), (64, 64), (130, 200)])
@pytest.mark.parametrize("kfast", [True, False])
@pytest.mark.parametrize("a", [1.0, -0.5])
def test_pieces(cuda, rows, k, kfast, a):
    x = values(rows * k, np.random.default_rng(rows + k)).reshape(rows, k)
    t = torch.from_numpy(x if kfast else x.T.copy()).to(cuda)
    got = pack(Operand("rk", (t, "rk" if kfast else "kr"), a=a), ["r"], ["k"], FMT_BF16X6, None)
    rest = a * x
    for piece in (got.hi, got.mid, got.lo):
        p = piece.view(torch.bfloat16).reshape(rows, got.Kp).double().cpu().numpy()
        want = bf16(rest)
        assert np.array_equal(p[:, :k], want)
        assert np.array_equal(np.signbit(p[:, :k])[want != 0], np.signbit(want)[want != 0])
        assert not p[:, k:].any()
        rest = rest - want
