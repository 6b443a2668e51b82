"""pcg_tc_gemm with fewer rows or columns than its output's sub-indices cover: only the elements that
the product reaches are cleared and written, in a launch whose K is split too."""
import pytest
import torch

from pycc_gb300 import _lib, tc
from pycc_gb300.tc import FMT_BF16, Operand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(40, 24), (33, 24), (40, 17), (33, 17)])
@pytest.mark.parametrize("order", ["rows inner", "columns inner"])
def test_part_of_the_output(cuda, M, N, order):
    gen = torch.Generator(device=cuda).manual_seed(M + N)
    # integers, exact in BF16 and in the sums
    ints = lambda *s: torch.randint(-4, 5, s, device=cuda, generator=gen).double()
    a, b = ints(M, 4096), ints(N, 4096)
    A = tc.pack(Operand("rk", (a, "rk")), ["r"], ["k"], FMT_BF16)
    B = tc.pack(Operand("ck", (b, "ck")), ["c"], ["k"], FMT_BF16)
    out = torch.full((24, 40) if order == "rows inner" else (40, 24), 7.0, dtype=torch.float64,
                     device=cuda)
    C = out.t() if order == "rows inner" else out           # [40 rows][24 columns]
    status = torch.zeros(4, dtype=torch.int32, device=cuda)
    tc.gemm(FMT_BF16, A, B, C, ["r"], ["c"], "rc", beta=0.0, status=status)
    want = torch.full_like(C, 7.0)
    want[:M, :N] = a @ b.t()
    assert int(status.abs().sum()) == 0
    assert torch.equal(C, want)
