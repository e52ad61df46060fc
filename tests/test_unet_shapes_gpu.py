"""The network's convolution, weight gradient and resampling kernels at the
volumes where their tiles go wrong first: one voxel per axis, lines just below,
at and above a tile's 128, partial tiles in every axis, against the FP64
oracle / torch.  Bars: BF16 outputs 4e-3 relative L2 (half a unit in the last
place is 2^-9), FP32 weight gradients 1e-5."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VOLUMES = [(1, 1, 1, 1), (7, 5, 3, 2), (16, 1, 9, 1), (62, 11, 5, 1), (127, 3, 2, 1), (128, 5, 3, 1), (129, 4, 2, 2),
           (260, 3, 2, 1)]
CHANNELS = [(16, 16), (48, 16), (16, 48), (64, 64), (96, 32), (32, 96)]


def P(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / max(np.linalg.norm(np.ravel(b)), 1e-30))


def _bf(a, dev):
    import torch
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float32), dtype=torch.bfloat16, device=dev).reshape(-1)


def _st(dev):
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


@pytest.mark.parametrize("X,Y,Z,B", VOLUMES)
@pytest.mark.parametrize("ci,co", CHANNELS)
def test_conv_and_wgrad_at_ragged_volumes(cuda, ci, co, X, Y, Z, B):
    import torch
    from oracle import unet_oracle as uo
    from omega_b200 import _native
    rng = np.random.default_rng(X * 100 + ci)
    x = uo.bf16(rng.normal(0, 1, (B, Z, Y, X, ci)))
    w = uo.bf16(rng.normal(0, 0.1, (27, co, ci)))
    b = rng.normal(0, 0.1, co).astype(np.float32)
    dz = uo.bf16(rng.normal(0, 1, (B, Z, Y, X, co)))
    mask = uo.bf16(rng.normal(0, 1, (B, Z, Y, X, co)))
    xt, wt, bt, dzt, mt = _bf(x, cuda), _bf(w, cuda), torch.tensor(b, device=cuda), _bf(dz, cuda), _bf(mask, cuda)
    ref = uo.conv3d(x, w, np.zeros(co))
    for bias, m, relu in ((bt, None, 1), (None, mt, 0), (bt, None, 0)):
        out = torch.full((B * Z * Y * X * co,), 7.0, dtype=torch.bfloat16, device=cuda)
        _native.call("omb_unet_conv_tc", ci, co, P(xt), P(wt), P(bias), P(out), P(m), relu, X, Y, Z, B, _st(cuda))
        want = ref + (b if bias is not None else 0.0)
        want = np.maximum(want, 0) if relu else want
        want = np.where(mask > 0, want, 0.0) if m is not None else want
        assert _rel(out.float().cpu().numpy().reshape(want.shape), want) < 4e-3
    dw = torch.zeros(27 * co * ci, device=cuda)
    _native.call("omb_unet_conv_wgrad", ci, co, P(xt), P(dzt), P(dw), X, Y, Z, B, _st(cuda))
    refw = uo.conv3d_wgrad(x, dz)
    assert _rel(dw.cpu().numpy().reshape(refw.shape), refw) < 1e-5
    flag = ctypes.c_int32(-1)
    _native.call("omb_unet_take_error", ctypes.byref(flag))
    assert flag.value == 0
