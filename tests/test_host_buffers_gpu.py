"""GEMVs through page-locked host buffers of the library and of others, whole and in parts, aligned and not, with sizes on both sides of what a copy kernel moves
(128 KB in, 256 KB out): the results of pageable buffers, and nothing written beside them."""
import ctypes as C

import numpy as np
import pytest

import pyre_b200 as pb

pytestmark = pytest.mark.gpu


def _gemv(ctx, W, x, t, y):
    ctx.check(pb.lib().pb_gemv(ctx.h, W.h, x.ctypes.data_as(C.c_void_p), C.c_int(t), y.ctypes.data_as(C.c_void_p)))


@pytest.mark.parametrize("owner", ["library", "other"])
@pytest.mark.parametrize("rows,t", [(4096, 1), (4096, 16), (4096, 17), (4099, 3), (515, 31)])
def test_page_locked_buffers(ctx, owner, rows, t):
    import torch
    cols, pad = 2048, 64
    W = pb.QMat.synth(ctx, pb.Q4_K, rows, cols, 0, 5)
    ref = np.empty((t, rows), np.float32)
    xs = np.random.default_rng(rows + t).standard_normal(t * cols).astype(np.float32)
    _gemv(ctx, W, xs, t, ref)
    n = t * (cols + rows) + 4 * pad
    buf = ctx.pinned_empty(n) if owner == "library" else torch.empty(n, pin_memory=True).numpy()
    for ox in (0, 1, 4):
        for oy in (0, 1, 4):
            buf[:] = -7.0
            x, y = buf[ox:ox + t * cols], buf[t * cols + pad + oy:t * cols + pad + oy + t * rows]
            x[:] = xs
            before = buf.copy()
            _gemv(ctx, W, x, t, y)
            assert np.array_equal(y.view(np.uint32), ref.ravel().view(np.uint32)), (ox, oy)
            y[:] = -7.0
            assert np.array_equal(buf.view(np.uint32), before.view(np.uint32)), (ox, oy)
    assert ctx.device_status() == 0
    W.free()


def test_a_buffer_that_was_freed_is_forgotten(ctx):
    """Page-locked results are given back and taken again while other calls use pageable memory at whatever addresses."""
    W = pb.QMat.synth(ctx, pb.Q8_0, 512, 512, 0, 6)
    x = np.random.default_rng(1).standard_normal((2, 512)).astype(np.float32)
    ref = W.matmul(x)
    for _ in range(20):
        y = ctx.pinned_empty((2, 512))
        _gemv(ctx, W, x, 2, y)
        assert np.array_equal(y.view(np.uint32), ref.view(np.uint32))
        del y
        z = np.empty((2, 512), np.float32)
        _gemv(ctx, W, x, 2, z)
        assert np.array_equal(z.view(np.uint32), ref.view(np.uint32))
    W.free()
