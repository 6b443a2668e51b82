"""The (T) energy kernel whose tiles come by TMA (pcg_triples_energy_pitched) against the FP64
kernel on the same partials, at nv around the tile edge and with and without f_ov.

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
    pitch = -(-nv // 4) * 4
    P = torch.full((3, 3, nv, nv, pitch), float("nan"), dtype=torch.float32, device=cuda)
    P[..., :nv] = rand(3, 3, nv, nv, nv).float()
    eoovv, t2, t1 = rand(no, no, nv, nv), rand(no, no, nv, nv), rand(no, nv)
    fov = None if canonical else rand(no, nv)
    eps = torch.cat([-1.0 - torch.rand(no, device=cuda, dtype=torch.float64),
                     1.0 + torch.rand(nv, device=cuda, dtype=torch.float64)])
    ijk = torch.tensor(trips, dtype=torch.int32, device=cuda)
    plen = int(_lib.load().pcg_triples_part_len(1, nv))
    part = torch.full((3, plen), float("nan"), dtype=torch.float64, device=cuda)
    status = torch.zeros(4, dtype=torch.int32, device=cuda)
    fp = None if fov is None else fov.data_ptr()
    ef, tf = (torch.full((no, no, nv, pitch), float("nan"), dtype=torch.float32, device=cuda)
              for _ in range(2))
    ef[..., :nv], tf[..., :nv] = eoovv.float(), t2.float()
    _lib.call("pcg_triples_energy_pitched", P.data_ptr(), pitch, ijk.data_ptr(), 3, eps.data_ptr(),
              ef.data_ptr(), t1.data_ptr(), tf.data_ptr(), fp, no, nv, part.data_ptr(),
              status.data_ptr(), _lib.stream_handle())
    P64 = P[..., :nv].double().contiguous()

    def ref():
        out = torch.empty((3, nv), dtype=torch.float64, device=cuda)
        _lib.call("pcg_triples_energy", 0, P64.data_ptr(), P64[:, 1].data_ptr(),
                  P64[:, 2].data_ptr(), 3 * nv ** 3, ijk.data_ptr(), 3, eps.data_ptr(),
                  eoovv.data_ptr(), t1.data_ptr(), t2.data_ptr(), fp, no, nv, out.data_ptr(),
                  _lib.stream_handle())
        return out.sum(1).cpu().numpy()
    got = part.sum(1).cpu().numpy()
    assert int(status.abs().sum()) == 0
    # magnitudes: W V products, six orderings with weights up to 3 + 2 * 9
    w = 3 * P64.abs().amax(dim=(1, 2, 3, 4)).cpu().numpy()
    d = 3 * float(eoovv.abs().max() * t1.abs().max())
    d += 0.0 if fov is None else 3 * float(t2.abs().max() * fov.abs().max())
    mag = 2 * (nv + 2) ** 3 / 6.0 * 60 * w * (w + d) / 6.0
    assert (np.abs(got - ref()) <= 64 * 2.0 ** -24 * mag).all()
