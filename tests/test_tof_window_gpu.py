"""TOF projections through the sliding window of bins: windows smaller than
the bin count (the ray moves through them), as large as it (an odd
number pads it), the series and the exponential form of the weights, both ray-driven
projectors, float and int64 backprojection, against the FP64 oracle (which
evaluates every bin of every element).  Bar: the projectors' own 1e-5
relative L2; the bins a window leaves out carry less than 2^-30 of an
element's weight."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-5
C = 2.99792458e11


def _options(projector, bins, fwhm, **attrs):
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(),
              dict(CONFIGS["pet_mini"], projector_type=projector, TOF_bins=bins, TOF_bins_used=bins, TOF_FWHM=fwhm,
                   TOF_width=255.0 / bins / (C / 2.), **attrs))
    o.addProjector()
    o.initProj()
    return o


@pytest.mark.parametrize("projector", [1, 4])
@pytest.mark.parametrize("bins,fwhm", [(3, 100e-12), (9, 60e-12), (15, 60e-12), (13, 400e-12),
                                       (15, 500e-12), (5, 30e-12)])
def test_windowed_tof_matches_oracle(cuda, projector, bins, fwhm):
    import torch
    o = _options(projector, bins, fwhm, use_64bit_atomics=bins == 9)
    g = orc.Geometry(o)
    fwd, bwd = (orc.forward, orc.backward) if projector == 1 else (orc.interp_forward, orc.interp_backward)
    rng = np.random.default_rng(bins)
    x = rng.uniform(0.2, 2.0, g.n_img).astype(np.float32)
    y = o.forwardProject(torch.from_numpy(x).to(cuda), 1).cpu().numpy()
    assert orc.rel_l2(y, fwd(g, x, 1)) < TOL
    m = rng.poisson(0.7, y.size).astype(np.float32)   # many bins, and whole rays, without counts
    img, sens = o.backwardProject(torch.from_numpy(m).to(cuda), 1, sens=True)
    ref, ref_s = bwd(g, m, 1, sens=True)
    assert orc.rel_l2(img.cpu().numpy(), ref) < TOL
    assert orc.rel_l2(sens.cpu().numpy(), ref_s) < TOL


@pytest.mark.parametrize("spacing", [200.0, 900.0])
def test_bins_far_from_the_image(cuda, spacing):
    """Bins out to 1.4 m beside a 180 mm image (sigma 3.3 mm, elements of up to
    4.1 mm: the series form) and out to 6.3 m.  The int64 backprojection keeps
    all of them, and what one adds far from its centre is 0, not 0 times
    infinity."""
    import torch
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(),
              dict(CONFIGS["pet_mini"], TOF_bins=15, TOF_bins_used=15, TOF_width=spacing / (C / 2.),
                   TOF_FWHM=3.3 * np.sqrt(8 * np.log(2.0)) * 2 / C, use_64bit_atomics=True, Nx=64, Ny=64, Nz=31))
    o.addProjector()
    o.initProj()
    g = orc.Geometry(o)
    rng = np.random.default_rng(5)
    m = rng.poisson(2.0, g.rays(1) * g.nbins).astype(np.float32)
    img, sens = o.backwardProject(torch.from_numpy(m).to(cuda), 1, sens=True)
    ref, ref_s = orc.backward(g, m, 1, sens=True)
    assert orc.rel_l2(img.cpu().numpy(), ref) < TOL
    assert orc.rel_l2(sens.cpu().numpy(), ref_s) < TOL


@pytest.mark.parametrize("projector", [1, 4])
def test_bins_in_pairs(cuda, projector):
    """Bins in close pairs 18 sigma apart: between two pairs the nearest bins
    are as far away as the ones a window of two would leave out.  (With a
    smallest weight below theirs the element still belongs to them.)"""
    import torch
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(),
              dict(CONFIGS["pet_mini"], projector_type=projector, TOF_bins=6, TOF_bins_used=6, TOF_width=30.0 / (C / 2.),
                   TOF_FWHM=5.0 * np.sqrt(8 * np.log(2.0)) * 2 / C, epps=1e-25))
    o.TOFCenter = np.array([0.0, 0.5, 90.0, 90.5, -90.0, -90.5], dtype=np.float32)
    o.sigma_x = 5.0
    o.addProjector()
    o.initProj()
    g = orc.Geometry(o)
    fwd, bwd = (orc.forward, orc.backward) if projector == 1 else (orc.interp_forward, orc.interp_backward)
    rng = np.random.default_rng(6)
    x = rng.uniform(0.2, 2.0, g.n_img).astype(np.float32)
    y = o.forwardProject(torch.from_numpy(x).to(cuda), 1).cpu().numpy()
    assert orc.rel_l2(y, fwd(g, x, 1)) < TOL
    m = rng.poisson(2.0, y.size).astype(np.float32)
    img, sens = o.backwardProject(torch.from_numpy(m).to(cuda), 1, sens=True)
    ref, ref_s = bwd(g, m, 1, sens=True)
    assert orc.rel_l2(img.cpu().numpy(), ref) < TOL
    assert orc.rel_l2(sens.cpu().numpy(), ref_s) < TOL
