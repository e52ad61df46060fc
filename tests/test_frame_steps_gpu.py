"""The frame-batched OSEM sub-iteration (frame-major, 4 and 8 frames per walk,
the EM update fused with the interleaved backprojection) against single
studies, and the PDHG dual step against FP64: sizes that are and are not
multiples of four, a buffer off a 16-byte boundary."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def P(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("frames", [3, 5, 9])
@pytest.mark.parametrize("shape", [(32, 32, 15), (33, 31, 7)])
def test_batched_osem_equals_single_studies(cuda, shape, frames):
    import torch
    from configs import CONFIGS, apply
    from omega_b200 import reconstruction as rec
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(), dict(CONFIGS["pet_mini"], Nx=shape[0], Ny=shape[1], Nz=shape[2]))
    o.addProjector()
    o.initProj()
    M, n = o.measurementCount(-1), int(o.N[0])
    g = torch.Generator(device=cuda).manual_seed(3)
    m = torch.poisson(torch.full((frames, M), 4.0, device=cuda), generator=g)
    x0 = torch.rand(frames, n, generator=g, device=cuda) + 0.5
    batch = rec.OSEMBatch(o, m, x0=x0.clone())
    got = batch.iterate(1)
    for f in range(frames):
        one = rec.OSEM(o, m[f].clone(), x0=x0[f].cpu().numpy())
        want = one.iterate(1)
        rel = float((got[f] - want).norm() / want.norm())
        assert rel < 1e-5, (f, rel)


@pytest.mark.parametrize("n,offset", [(4096, 0), (4097, 0), (4096, 1), (3, 0), (1, 0)])
def test_dual_step(cuda, n, offset):
    import torch
    from omega_b200 import _native
    g = torch.Generator(device=cuda).manual_seed(n)
    t = lambda: torch.randn(n + offset, generator=g, device=cuda)[offset:]  # noqa: E731
    p, fp, y = t(), t(), t()
    want = (p.double() + 0.7 * (fp.double() - y.double())) / 1.7
    _native.call("omb_pdhg_dual", P(p), P(fp), P(y), n, 0.7, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert torch.allclose(p.double(), want, atol=1e-6, rtol=1e-5)
