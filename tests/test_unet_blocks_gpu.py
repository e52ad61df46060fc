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
