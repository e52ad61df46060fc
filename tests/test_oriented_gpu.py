"""Ray-driven projections whose rays along x go through the y-fastest copy of
the image: grids that are not square (the copy's strides differ), odd sizes,
both projectors, TOF, BF16 reads, float and int64 backprojection, the subset
types whose neighbouring rays are neighbours on the detector and one whose
rays are not, against the FP64 oracle.  Bar: the projectors' own 1e-5 relative
L2."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _options(**attrs):
    from configs import CONFIGS, apply
    from omega_b200.projector import proj
    o = apply(proj.projectorClass(), dict(CONFIGS["pet_mini"], **attrs))
    o.addProjector()
    o.initProj()
    return o


@pytest.mark.parametrize("projector", [1, 4])
@pytest.mark.parametrize("shape", [(33, 45, 15), (61, 32, 7), (40, 40, 15)])
@pytest.mark.parametrize("extra", [{}, {"use_64bit_atomics": True}, {"imageReadPrecision": "bf16"},
                                   {"subsetType": 2}, {"subsetType": 4}, {"subsetType": 1},
                                   {"TOF_bins": 5, "TOF_bins_used": 5, "TOF_FWHM": 200e-12,
                                    "TOF_width": 50.0 / (2.99792458e11 / 2.)}])
def test_oriented_projections_match_oracle(cuda, projector, shape, extra):
    import torch
    o = _options(projector_type=projector, Nx=shape[0], Ny=shape[1], Nz=shape[2], FOVa_x=170., FOVa_y=150., **extra)
    g = orc.Geometry(o)
    fwd, bwd = (orc.forward, orc.backward) if projector == 1 else (orc.interp_forward, orc.interp_backward)
    rng = np.random.default_rng(shape[0])
    x = rng.uniform(0.2, 2.0, g.n_img).astype(np.float32)
    if "imageReadPrecision" in extra:
        x = torch.from_numpy(x).bfloat16().float().numpy()   # what the reads round to
    for s in (0, g.n_subsets - 1):
        y = o.forwardProject(torch.from_numpy(x).to(cuda), s).cpu().numpy()
        assert orc.rel_l2(y, fwd(g, x, s)) < TOL, s
        m = rng.poisson(1.5, y.size).astype(np.float32)
        img = o.backwardProject(torch.from_numpy(m).to(cuda), s).cpu().numpy()
        assert orc.rel_l2(img, bwd(g, m, s)) < TOL, s
        if "use_64bit_atomics" in extra:
            again = o.backwardProject(torch.from_numpy(m).to(cuda), s).cpu().numpy()
            assert np.array_equal(img.view(np.uint32), again.view(np.uint32))


def test_oriented_projections_in_a_graph(cuda):
    """A captured call (which takes no copy) replays with the eager call's
    result, also after eager calls of other images."""
    import torch
    o = _options(Nx=33, Ny=45, FOVa_x=170., FOVa_y=150.)
    n = int(o.N[0])
    gen = torch.Generator(device=cuda).manual_seed(1)
    x = torch.rand(n, generator=gen, device=cuda)
    want = o.forwardProject(x, 0).clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        o.forwardProject(x, 0)
    torch.cuda.current_stream().wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = o.forwardProject(x, 0)
    for _ in range(3):
        o.forwardProject(torch.rand(n, device=cuda), 0)
        y.zero_()
        graph.replay()
        assert torch.equal(y, want)
    del graph


@pytest.mark.parametrize("projector", [1, 4])
def test_captured_projections_hold_no_memory_nodes(cuda, projector):
    """A graph with memory allocation nodes can be neither cloned nor
    instantiated twice at once; these can, and both instances compute the
    projections."""
    import ctypes

    import torch
    rt = ctypes.CDLL("libcudart.so.12")
    o = _options(Nx=33, Ny=45, FOVa_x=170., FOVa_y=150., projector_type=projector)
    gen = torch.Generator(device=cuda).manual_seed(2)
    x = torch.rand(int(o.N[0]), generator=gen, device=cuda)
    want_y = o.forwardProject(x, 0).clone()
    want_b = o.backwardProject(want_y, 0).clone()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        y = o.forwardProject(x, 0)
        b = o.backwardProject(y, 0)
    raw = ctypes.c_void_p(graph.raw_cuda_graph())
    n = ctypes.c_size_t(0)
    assert rt.cudaGraphGetNodes(raw, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(raw, nodes, ctypes.byref(n)) == 0
    for node in nodes:
        kind = ctypes.c_int(-1)
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        assert kind.value not in (10, 11)   # memory allocation, memory free
    clone = ctypes.c_void_p()
    assert rt.cudaGraphClone(ctypes.byref(clone), raw) == 0
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    execs = []
    for g in (raw, clone):
        e = ctypes.c_void_p()
        assert rt.cudaGraphInstantiate(ctypes.byref(e), g, ctypes.c_ulonglong(0)) == 0
        execs.append(e)
    for e in execs:
        y.zero_()
        b.zero_()
        assert rt.cudaGraphLaunch(e, stream) == 0
        torch.cuda.synchronize()
        assert float((y - want_y).norm() / want_y.norm()) < 1e-6
        assert float((b - want_b).norm() / want_b.norm()) < 1e-6
    for e in execs:
        assert rt.cudaGraphExecDestroy(e) == 0
    assert rt.cudaGraphDestroy(clone) == 0
