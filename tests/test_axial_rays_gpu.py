"""Rays that run along z (end points equal in x and apart by less than 1e-6 in
y, or the other way round), inside and outside the image and ending inside and
outside its slices, among ordinary ones: list-mode events, type 1, against the
FP64 oracle.  Where x alone is equal the first voxel takes the ray, as in the
reference's kernels.  Bar: the projector's own 1e-5 relative L2."""
import ctypes

import numpy as np
import pytest

from conftest import listmode_events
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _options(**attrs):
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    _, ev, _ = listmode_events("pet_mini", 200, 3)
    rng = np.random.default_rng(4)
    along = []
    for k in range(120):
        u, v = rng.uniform(-100, 100, 2) * (1 if k % 5 else 0)   # the image is 180 mm wide; some along its middle
        z = np.sort(rng.uniform(-30, 30, 2))[::1 if k % 2 else -1] if k % 3 else rng.choice([-25, 25]) * np.array([1, -1])
        # (a difference this small survives only around 0)
        tiny = rng.choice([1e-30, 2e-14, 3e-7]) * rng.choice([-1, 1])
        along.append([u, 0.0, z[0], u, tiny, z[1]] if k % 4 else [0.0, v, z[0], tiny, v, z[1]])
    ev = np.concatenate([ev, np.array(along).T], 1)[:, rng.permutation(320)]
    o = apply(proj.projectorClass(), dict(CONFIGS["pet_mini"], subsets=1, **attrs))
    o.SinM = np.zeros(ev.shape[1], dtype=np.float32)
    o.x = np.asfortranarray(ev.astype(np.float32))
    o.addProjector()
    o.initProj()
    return o


@pytest.mark.parametrize("extra", [{}, {"use_64bit_atomics": True}, {"imageReadPrecision": "bf16"},
                                   {"Nx": 7, "Ny": 1}])
def test_rays_along_z_match_oracle(cuda, extra):
    import torch
    from omega_b200 import _native
    o = _options(**extra)
    g = orc.Geometry(o)
    rng = np.random.default_rng(5)
    x = rng.uniform(0.2, 2.0, g.n_img).astype(np.float32)
    if "imageReadPrecision" in extra:
        x = torch.from_numpy(x).bfloat16().float().numpy()
    ref = orc.forward(g, x, 0)
    m = rng.poisson(1.5, ref.size).astype(np.float32)
    ref_b, ref_s = orc.backward(g, m, 0, sens=True)
    for steps in (1, 2, 4):
        o.tuning = {"siddon_fp_steps": steps}
        y = o.forwardProject(torch.from_numpy(x).to(cuda), 0).cpu().numpy()
        assert np.abs(y - ref).max() < TOL * np.abs(ref).max(), steps
    img, sens = o.backwardProject(torch.from_numpy(m).to(cuda), 0, sens=True)
    assert orc.rel_l2(img.cpu().numpy(), ref_b) < TOL
    assert orc.rel_l2(sens.cpu().numpy(), ref_s) < TOL
    assert orc.rel_l2(o.backwardProject(torch.from_numpy(m).to(cuda), 0).cpu().numpy(), ref_b) < TOL
    if not extra:
        frames, n = 5, g.n_img
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        X = torch.from_numpy(np.tile(x, (frames, 1))).to(cuda)
        M = torch.from_numpy(np.tile(m, (frames, 1))).to(cuda)
        Y, B = torch.empty(frames, ref.size, device=cuda), torch.empty(frames, n, device=cuda)
        P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        _native.call("omb_forward_frames", o._handle, 0, frames, P(X), n, P(Y), ref.size, st)
        _native.call("omb_backward_frames", o._handle, 0, frames, P(M), ref.size, P(B), n, st)
        for f in range(frames):
            assert orc.rel_l2(Y[f].cpu().numpy(), ref) < TOL
            assert orc.rel_l2(B[f].cpu().numpy(), ref_b) < TOL


def test_tof_leaves_them_out(cuda):
    """TOF data has no list-mode form here; sinogram bins set to such pairs add
    nothing, and the bins around them are what they are."""
    import torch
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(), dict(CONFIGS["pet_mini"], TOF_bins=5, TOF_bins_used=5, TOF_FWHM=120e-12,
                                          TOF_width=40.0 / (2.99792458e11 / 2.)))
    o.addProjector()
    xy = np.array(o.x, dtype=np.float32).reshape(-1, 4)
    here = np.arange(len(xy)) % 9 == 0
    xy[here] = np.stack([[u, 0.0, u, 2e-14] for u in np.linspace(-100, 100, here.sum())])
    o.x = xy.ravel()
    z = np.array(o.z, dtype=np.float32).reshape(-1, 2)
    z[z[:, 0] != z[:, 1]] = [-40.0, 40.0]   # through all slices
    o.z = z.ravel()
    o.initProj()
    g = orc.Geometry(o)
    n = int(o.nMeas[1])
    oblique = np.repeat(z[:n, 0] != z[:n, 1], len(xy))   # (where the slices are equal the end points coincide)
    skip, keep = (np.tile(np.tile(here == v, n) & oblique, 5) for v in (True, False))
    assert skip.any() and keep.any()
    x = np.random.default_rng(7).uniform(0.2, 2.0, g.n_img).astype(np.float32)
    y = o.forwardProject(torch.from_numpy(x).to(cuda), 0).cpu().numpy()
    ref = orc.forward(g, x, 0)
    assert np.all(y[skip] == 0)
    assert orc.rel_l2(y[keep], ref[keep]) < TOL
    m = np.where(skip, 3.0, 0.0).astype(np.float32)
    assert not o.backwardProject(torch.from_numpy(m).to(cuda), 0).any()
    m = np.where(skip | keep, 1.0, 0.0).astype(np.float32)
    img = o.backwardProject(torch.from_numpy(m).to(cuda), 0).cpu().numpy()
    assert orc.rel_l2(img, orc.backward(g, np.where(keep, 1.0, 0.0), 0)) < TOL
