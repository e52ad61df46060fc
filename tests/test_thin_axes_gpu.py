"""Images one voxel thick along an axis, with rays oblique to it: both
ray-driven projectors, PET and cone-beam CT, TOF, BF16 reads, float and int64
backprojection, against the FP64 oracle.  Bar: the projectors' own 1e-5
relative L2, except for float sums into fewer than 100 voxels: every ray of the
subset adds to each of them, and n FP32 additions of one sign round by up to n *
2^-24 of their sum (the int64 sums of the same rays keep the 1e-5)."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-5
TOF = {"TOF_bins": 5, "TOF_bins_used": 5, "TOF_FWHM": 200e-12, "TOF_width": 50.0 / (2.99792458e11 / 2.)}


def _options(name, shape, **attrs):
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(), dict(CONFIGS[name], Nx=shape[0], Ny=shape[1], Nz=shape[2], **attrs))
    o.addProjector()
    o.initProj()
    return o


@pytest.mark.parametrize("shape", [(32, 32, 1), (33, 45, 1), (1, 32, 15), (32, 1, 15), (33, 1, 1), (1, 1, 1)])
@pytest.mark.parametrize("name,extra", [("pet_mini", {}), ("pet_mini", TOF), ("pet_mini", {"use_64bit_atomics": True}),
                                        ("pet_mini4", {}), ("pet_mini4", TOF),
                                        ("pet_mini4", {"use_64bit_atomics": True}),
                                        ("pet_mini4", {"imageReadPrecision": "bf16"}),
                                        ("pet_mini4", dict(TOF, imageReadPrecision="bf16")),
                                        ("ct_mini", {}), ("ct_mini4", {}), ("ct_mini4", {"imageReadPrecision": "bf16"})])
def test_thin_axes_match_oracle(cuda, name, extra, shape):
    import torch
    o = _options(name, shape, **extra)
    g = orc.Geometry(o)
    fwd, bwd = (orc.interp_forward, orc.interp_backward) if name.endswith("4") else (orc.forward, orc.backward)
    if name == "ct_mini4":
        bwd = orc.interp_ct_backward
    rng = np.random.default_rng(shape[0])
    x = rng.uniform(0.2, 2.0, g.n_img).astype(np.float32)
    if "imageReadPrecision" in extra:
        x = torch.from_numpy(x).bfloat16().float().numpy()   # what the reads round to
    for s in (0, g.n_subsets - 1):
        y = o.forwardProject(torch.from_numpy(x).to(cuda), s).cpu().numpy()
        assert orc.rel_l2(y, fwd(g, x, s)) < TOL, s
        m = rng.poisson(1.5, y.size).astype(np.float32)
        img = o.backwardProject(torch.from_numpy(m).to(cuda), s).cpu().numpy()
        few = g.n_img < 100 and "use_64bit_atomics" not in extra
        assert orc.rel_l2(img, bwd(g, m, s)) < (max(TOL, g.rays(s) * 2.0 ** -24) if few else TOL), s
