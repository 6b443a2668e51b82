"""The (T) energy kernel for FP32 partials without a pitch (pcg_triples_energy, fp32 = 1), which
callers of the C interface use, against the FP64 kernel on the same partials.

Tolerance: each of the nv^3 / 6 terms carries about thirty FP32 roundings of sums of at most eight
products, and terms of both signs add up: 64 2^-24 of the sum of the terms' magnitudes, which the
partials' and integrals' magnitudes bound.
"""
import numpy as np
import pytest
import torch

from pycc_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 3, 8, 9, 16, 23, 40])
@pytest.mark.parametrize("canonical", [True, False])
def test_energy(cuda, nv, canonical):
    no, trips = 3, [(2, 1, 0), (2, 2, 1), (1, 1, 1)]
    gen = torch.Generator(device=cuda).manual_seed(nv)
    rand = lambda *s: torch.randn(s, dtype=torch.float64, device=cuda, generator=gen).float().double()
    P, eoovv, t2, t1 = rand(3, 3, nv, nv, nv), rand(no, no, nv, nv), rand(no, no, nv, nv), rand(no, nv)
    fov = None if canonical else rand(no, nv)
    eps = torch.cat([-1.0 - torch.rand(no, device=cuda, dtype=torch.float64),
                     1.0 + torch.rand(nv, device=cuda, dtype=torch.float64)])
    ijk = torch.tensor(trips, dtype=torch.int32, device=cuda)

    def energy(fp32):
        dt = torch.float32 if fp32 else torch.float64
        p, e, t = P.to(dt), eoovv.to(dt), t2.to(dt)
        plen = int(_lib.load().pcg_triples_part_len(fp32, nv))
        part = torch.full((3, plen), float("nan"), dtype=torch.float64, device=cuda)
        _lib.call("pcg_triples_energy", fp32, p.data_ptr(), p[:, 1].data_ptr(), p[:, 2].data_ptr(),
                  3 * nv ** 3, ijk.data_ptr(), 3, eps.data_ptr(), e.data_ptr(), t1.data_ptr(),
                  t.data_ptr(), None if fov is None else fov.data_ptr(), no, nv, part.data_ptr(),
                  _lib.stream_handle())
        return part.sum(1).cpu().numpy()
    # magnitudes: W V products, six orderings with weights up to 3 + 2 * 9
    w = 3 * P.abs().amax(dim=(1, 2, 3, 4)).cpu().numpy()
    d = 3 * float(eoovv.abs().max() * t1.abs().max())
    d += 0.0 if fov is None else 3 * float(t2.abs().max() * fov.abs().max())
    mag = 2 * (nv + 2) ** 3 / 6.0 * 60 * w * (w + d) / 6.0
    assert (np.abs(energy(1) - energy(0)) <= 64 * 2.0 ** -24 * mag).all()
