"""Calls after a failed one: an error is reported by the call that met it and by no other."""
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
