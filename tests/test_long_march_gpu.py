"""Type-4 marches of about a million samples per ray that drift across a voxel
of a nearly constant axis (each step below 1e-6 voxels), against the FP64
oracle.  Bar: a sum of n FP32 terms of one sign rounds by up to n * 2^-24 of
itself."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("read", ["fp32", "bf16"])
@pytest.mark.parametrize("axis", ["x", "y"])
def test_long_marches_match_oracle(cuda, axis, read):
    import torch
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    n = 1_200_000
    # texel coordinates of the transverse axis and of z at the two ends of the ray, scanner length 300 mm: the march
    # covers the middle 180 mm
    ends = [((10.3, 10.3), (0.6, -0.4)), ((10.3, 10.3), (-0.4, 0.6)), ((0.6, -0.4), (7.2, 7.2)),
            ((30.4, 31.4), (7.0, 7.0)), ((10.0, 10.9), (13.5, 14.4)), ((16.0, 16.0), (7.0, 7.0))]
    d = dict(CONFIGS["pet_mini"], projector_type=4, subsets=1, dL=180.0 / 5.625 / n, imageReadPrecision=read)
    ev = []
    for (u0, u1), (z0, z1) in ends:
        grow = 300.0 / 180.0   # ends of the scanner from ends of the image
        mu, du, mz, dz = (u0 + u1) / 2, (u1 - u0) / 2 * grow, (z0 + z1) / 2, (z1 - z0) / 2 * grow
        u = [(mu + k * du + 0.5) * 5.625 - 90 for k in (-1, 1)]
        z = [(mz + k * dz + 0.5) * 34 / 15 - 17 for k in (-1, 1)]
        ev.append([-150, u[0], z[0], 150, u[1], z[1]] if axis == "x" else [u[0], -150, z[0], u[1], 150, z[1]])
    o = apply(proj.projectorClass(), d)
    o.SinM = np.zeros(len(ev), dtype=np.float32)
    o.x = np.asfortranarray(np.array(ev, dtype=np.float32).T)
    o.addProjector()
    o.initProj()
    g = orc.Geometry(o)
    x = np.random.default_rng(1).uniform(0.5, 1.5, g.n_img).astype(np.float32)
    if read == "bf16":
        x = torch.from_numpy(x).bfloat16().float().numpy()
    y = o.forwardProject(torch.from_numpy(x).to(cuda), 0).cpu().numpy()
    ref = orc.interp_forward(g, x, 0)
    assert np.all(ref > 0)
    assert np.all(np.abs(y - ref) < n * 2.0 ** -24 * ref)
