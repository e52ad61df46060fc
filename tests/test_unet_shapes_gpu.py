"""The network's convolution, weight gradient and resampling kernels at the
volumes where their tiles go wrong first: one voxel per axis, lines just below,
at and above a tile's 128, partial tiles, against the FP64 oracle / torch.
(Volumes this small take one block of one line and one plane per thread block;
test_unet_blocks_gpu.py has the larger ones.)  Bars: BF16 outputs 4e-3 relative L2 (half a unit in the last
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


@pytest.mark.parametrize("c,offset", [(16, 0), (32, 0), (24, 0), (12, 0), (16, 1)])
def test_resampling_kernels(cuda, c, offset):
    """8 channels per thread (multiples of 8, aligned) and element by element
    (12 channels; a tensor that starts 2 bytes off)."""
    import torch
    from omega_b200 import _native
    X, Y, Z, B, cs = 6, 10, 4, 2, 16 if c % 8 == 0 else 4
    g = torch.Generator(device=cuda).manual_seed(c)

    def t(*shape):
        n = int(np.prod(shape))
        buf = torch.randn(n + offset, generator=g, device=cuda).bfloat16()
        return buf[offset:].view(*shape)

    full, half = t(B, Z, Y, X, c), t(B, Z // 2, Y // 2, X // 2, c)
    out = t(B, Z // 2, Y // 2, X // 2, c)
    _native.call("omb_unet_avgpool", P(full), P(out), X, Y, Z, B, c, 0, _st(cuda))
    pool = full.float().view(B, Z // 2, 2, Y // 2, 2, X // 2, 2, c).mean((2, 4, 6))
    assert torch.allclose(out.float(), pool, atol=1e-2, rtol=1e-2)
    up = lambda v: v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)  # noqa: E731
    din = full.clone() if offset == 0 else t(B, Z, Y, X, c)
    want = din.float() + 0.125 * up(half.float())
    _native.call("omb_unet_avgpool", P(half), P(din), X, Y, Z, B, c, 1, _st(cuda))
    assert torch.allclose(din.float(), want, atol=2e-2, rtol=1e-2)
    skip, cat = t(B, Z, Y, X, cs), t(B, Z, Y, X, c + cs)
    _native.call("omb_unet_up_concat", P(half), P(skip), P(cat), X, Y, Z, B, c, cs, _st(cuda))
    assert torch.equal(cat, torch.cat([up(half), skip], -1))
    dlow, dskip = t(B, Z // 2, Y // 2, X // 2, c), t(B, Z, Y, X, cs)
    want_skip = dskip.float() + cat[..., c:].float()
    _native.call("omb_unet_up_concat_bwd", P(cat), P(dlow), P(dskip), X, Y, Z, B, c, cs, _st(cuda))
    want_low = cat[..., :c].float().view(B, Z // 2, 2, Y // 2, 2, X // 2, 2, c).sum((2, 4, 6))
    assert torch.allclose(dlow.float(), want_low, atol=5e-2, rtol=1e-2)
    assert torch.allclose(dskip.float(), want_skip, atol=3e-2, rtol=1e-2)
    d = t(B, Z, Y, X, c)
    want = torch.where(full.float() > 0, d, torch.zeros_like(d))
    _native.call("omb_unet_relu_mask", P(d), P(full), d.numel(), _st(cuda))
    assert torch.equal(d, want)
