"""Calls after a failed or an awkward one: an error is reported by the call that met it and
by no other, choosing a launch shape asks the device for nothing, and the launch counter
counts every entry point's kernels."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def step(ctx, cells):
    out = np.empty_like(cells)
    ctx.upload(cells)
    rc, dt = ctx.prepare(0, 0.0, 0, True)
    rc2, moved = ctx.advance(0, dt, dt)
    ctx.download(out)
    return rc, rc2, moved, out.tobytes()


def test_failed_allocation_leaves_other_calls_alone(wr, gpu):
    """A context larger than any device is refused; what is called next, on a context that was
    there before, on a new one, and for gradients, works."""
    from warp_reactor_gb300 import diff
    cells = wr.make_grid(2)
    with wr.Context(len(cells)) as ctx:
        want = step(ctx, cells)
        assert want[:3] == (wr.SUCCESS, wr.SUCCESS, len(cells))
        with pytest.raises(wr.WarpReactorError):
            wr.Context(2**31 - 1)
        assert step(ctx, cells) == want
        with pytest.raises(wr.WarpReactorError):
            diff.DiffMap(2**31 - 1)
        assert step(ctx, cells) == want
    with pytest.raises(wr.WarpReactorError):
        wr.Context(2**31 - 1)
    with wr.Context(len(cells)) as ctx:
        assert step(ctx, cells) == want

def test_choosing_a_shape_during_a_capture(wr, gpu):
    """A program may choose a context's launch shape while it captures a stream of its own."""
    try:
        cudart = ctypes.CDLL("libcudart.so")
    except OSError:
        from warp_reactor_gb300 import build
        cudart = ctypes.CDLL(os.path.join(build._cuda_home(), "lib64", "libcudart.so"))
    cells = wr.make_grid(2)
    with wr.Context(len(cells)) as ctx:
        want = step(ctx, cells)
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    with wr.Context(len(cells)) as ctx:
        assert cudart.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0  # non-blocking
        assert cudart.cudaStreamBeginCapture(stream, 1) == 0                   # this thread's calls
        ctx.set_variant(2)
        assert cudart.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
        assert step(ctx, cells) == want
    assert cudart.cudaGraphDestroy(graph) == 0 and cudart.cudaStreamDestroy(stream) == 0


def test_launch_count(wr, gpu):
    """wr_kernel_launch_count over the entry points that launch kernels of their own."""
    import torch
    from warp_reactor_gb300 import diff
    cells = wr.make_grid(2)
    with wr.Context(len(cells), 0, wr.MATH_PORTABLE) as ctx:
        ctx.upload(cells)
        _, dt = ctx.prepare(0, 0.0, 0, True)
    records = torch.from_numpy(cells.view(np.uint8).copy()).cuda()
    q = torch.empty(len(cells), 15, dtype=torch.float64, device="cuda")
    p = torch.empty(diff.num_multipliers(), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f, moved = wr.lib().wr_advance_cells_noalloc, ctypes.c_int()
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double,
                  ctypes.POINTER(ctypes.c_int)]
    with diff.DiffMap(len(cells), max_outer_steps=1) as dmap:
        before = wr.kernel_launch_count()
        dmap.forward(records, None, None, [dt], False, q)
        dmap.backward(torch.ones_like(q), torch.empty_like(q), p)
        assert wr.kernel_launch_count() - before == 4  # multipliers, forward; backward, their sum
    before = wr.kernel_launch_count()
    assert f(records.data_ptr(), len(cells), 0, dt, dt, ctypes.byref(moved)) == wr.SUCCESS
    assert wr.kernel_launch_count() - before == 5      # unpack, queue, advance, commit, pack
