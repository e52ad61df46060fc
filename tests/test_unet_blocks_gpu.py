"""The network's convolutions where a thread block works through several blocks
of voxels and several launches share an SM's tensor memory."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def P(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _inputs(dev, ci, co, n, seed):
    import torch
    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev)  # noqa: E731
    return rnd(n * ci).bfloat16(), (rnd(27 * co * ci) * 0.1).bfloat16(), rnd(co) * 0.1


def test_launches_that_share_tensor_memory(cuda):
    """Short launches along lines of 65 to 128 voxels and of other shapes, on
    two streams: an SM hands tensor memory from one launch's block to the next
    launch's.  A sum has a fixed order, so every result equals that of the
    launch alone, bit for bit."""
    import torch
    from omega_b200 import _native
    cases = []
    for k, (ci, co, X, Y, Z, B) in enumerate([(16, 16, 128, 9, 7, 8), (32, 32, 62, 11, 9, 8), (48, 16, 100, 5, 6, 8),
                                              (64, 64, 33, 17, 8, 4), (16, 48, 128, 6, 5, 8)]):
        x, w, b = _inputs(cuda, ci, co, X * Y * Z * B, k)

        def launch(out, stream, x=x, w=w, b=b, args=(ci, co, X, Y, Z, B)):
            c, o, X, Y, Z, B = args
            _native.call("omb_unet_conv_tc", c, o, P(x), P(w), P(b), P(out), None, 1, X, Y, Z, B,
                         ctypes.c_void_p(stream.cuda_stream))
        alone = torch.empty(X * Y * Z * B * co, dtype=torch.bfloat16, device=cuda)
        launch(alone, torch.cuda.current_stream())
        torch.cuda.synchronize()
        cases.append((launch, alone, [torch.empty_like(alone) for _ in range(2)]))
    orders = [(torch.cuda.Stream(), cases), (torch.cuda.Stream(), cases[::-1])]
    for rep in range(20):
        for i, (stream, order) in enumerate(orders):
            for launch, _, outs in order:
                launch(outs[i], stream)
        torch.cuda.synchronize()
        for _, alone, outs in cases:
            for out in outs:
                assert torch.equal(out, alone), rep
    flag = ctypes.c_int32(-1)
    _native.call("omb_unet_take_error", ctypes.byref(flag))
    assert flag.value == 0


def _shifts(x):
    """The 27 neighbours of every voxel of x [B][Z][Y][X][C], zeros outside."""
    import torch
    B, Z, Y, X, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    for tap in range(27):
        dz, dy, dx = tap // 9, tap // 3 % 3, tap % 3
        yield tap, xp[:, dz:dz + Z, dy:dy + Y, dx:dx + X]


# On 148 SMs: several lines (TY 2 to 5) and planes (TZ 2 to 8) per block that do not divide the axes and up to 7
# blocks per thread block (61 x 63 x 31, 64 x 64 x 32); lines of 65 to 128 voxels with several planes (TZ 3 to 7) and
# lines (YS 6 to 11) per block, one (125) and up to 3 (67) blocks per thread block; weight gradients of 12 to 240
# stages per thread block, with two and three stages in flight, below and past the 32 to 85 after which sums go to
# memory.
BLOCKS = [(61, 63, 31, 4), (64, 64, 32, 4), (125, 67, 33, 2), (67, 11, 7, 150), (70, 23, 11, 90)]


@pytest.mark.parametrize("X,Y,Z,B", BLOCKS)
@pytest.mark.parametrize("ci,co", [(16, 16), (32, 32), (48, 16), (16, 48), (64, 64), (96, 32), (32, 96)])
def test_several_blocks_per_thread_block(cuda, ci, co, X, Y, Z, B):
    """Every output voxel of the convolution, and the weight gradient, against
    FP64.  Bars: a BF16 output is off by half a unit (2^-9 of it) and what FP32
    sums of up to 2592 products move it across a tie (below 1e-3 of the outputs'
    root mean square); a weight gradient's FP32 sums of up to 8192 voxels at a
    time stay within 1e-5 of its norm, any value within 1e-4 of its root mean
    square."""
    import torch
    from omega_b200 import _native
    st = ctypes.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)
    n = X * Y * Z * B
    x, w, b = _inputs(cuda, ci, co, n, X + ci)
    dz = torch.randn(n * co, generator=torch.Generator(device=cuda).manual_seed(co), device=cuda).bfloat16()
    out = torch.full((n * co,), 7.0, dtype=torch.bfloat16, device=cuda)
    _native.call("omb_unet_conv_tc", ci, co, P(x), P(w), P(b), P(out), None, 0, X, Y, Z, B, st)
    dw = torch.zeros(27 * co * ci, device=cuda)
    _native.call("omb_unet_conv_wgrad", ci, co, P(x), P(dz), P(dw), X, Y, Z, B, st)
    xd, wd = x.double().view(B, Z, Y, X, ci), w.double().view(27, co, ci)
    ref = b.double().expand(n, co).clone()
    refw = torch.empty_like(wd)
    dzt = dz.double().view(n, co).T.contiguous()
    for tap, xs in _shifts(xd):
        xs = xs.reshape(n, ci)
        ref.addmm_(xs, wd[tap].T)
        refw[tap] = dzt @ xs
    rms = float(ref.square().mean().sqrt())
    assert bool(((out.double().view(n, co) - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3 * rms).all())
    d = dw.double().view_as(refw) - refw
    assert float(d.norm() / refw.norm()) < 1e-5
    assert float(d.abs().max()) < 1e-4 * float(refw.square().mean().sqrt())
    flag = ctypes.c_int32(-1)
    _native.call("omb_unet_take_error", ctypes.byref(flag))
    assert flag.value == 0
