"""A rejected attempt of the cooperative advance retries from the kept Jacobian and
right-hand side; where cells of one warp disagree (one accepted, one rejected, or a
group without a cell), the program runs again for all of them.  The lane-per-cell
advance keeps the Jacobian per cell, so both give the same bits and counters."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("math", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 33])
def test_retries_equal_lane_per_cell(wr, gpu, n, math):
    """Unlike cells, alone in a warp, in pairs, and with an odd one left over, at 8, 16
    and 32 lanes per cell against the lane-per-cell advance: no tolerance."""
    start = wr.make_batch_grid(3, n)

    def burn(variant):
        cells = start.copy()
        with wr.Context(n, 0, math) as ctx:
            ctx.set_variant(variant)
            ctx.upload(cells)
            rc, cgs = ctx.run(True)
            ctx.download(cells)
        return rc, cgs, cells

    rc, cgs, want = burn(2)
    assert want["stats"]["internal_steps"].sum() > want["stats"]["accepted_steps"].sum()  # there are rejections
    for variant in (5, 6, 7):
        got = burn(variant)
        assert got[:2] == (rc, cgs)
        assert got[2].tobytes() == want.tobytes(), variant
