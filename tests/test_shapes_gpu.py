"""The launch shapes that a context or a call picks by its number of cells, each reached on
purpose (sizes follow the device's SM count) and compared with another implementation:
the CPU oracle, the lane-per-cell advance, the reference kernel's recorded states."""
import ctypes
import os
import time

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sms(gpu):
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("math", [0, 1])
@pytest.mark.parametrize("tiles", [lambda sms: sms // 5, lambda sms: sms // 4, lambda sms: sms // 4 + 1,
                                   lambda sms: sms // 2, lambda sms: sms // 2 + 1, lambda sms: sms + 3],
                         ids=["four_blocks", "four_to_two", "two_blocks", "two_blocks_most", "one_block", "queue"])
def test_cta32_shapes(wr, gpu, sms, oracle_port, tiles, math):
    """The structured policy on clusters of four blocks, of two, and on one block per tile
    (more tiles than SMs: blocks take a second one), the last tile ragged: three outer
    steps of unlike cells against the oracle (portable math) and, in both maths, against
    the same tiles as grids of their own."""
    n = 32 * tiles(sms) - 13
    cells = wr.make_batch_grid(3, n)

    def steps(part, dts=None):
        out, taken, t = part.copy(), [], 0.0
        with wr.Context(len(out), 0, math) as ctx:
            ctx.upload(out)
            for k in range(3):
                ctx.set_policy(wr.POLICY_GRIDWIDE_INDEPENDENT)  # the two policies' prepare is the same
                rc, dt = ctx.prepare(k, t, k, True)
                assert rc == wr.SUCCESS
                dt = dt if dts is None else dts[k]
                ctx.set_policy(wr.POLICY_GRIDWIDE_CTA32)
                rc, moved = ctx.advance(k, t + dt, dt)
                assert rc == wr.SUCCESS and moved == len(out)
                taken.append(dt)
                t += dt
            ctx.download(out)
        return out, taken

    got, dts = steps(cells)
    assert got["stats"]["internal_steps"].sum() > got["stats"]["accepted_steps"].sum()  # rejected trials
    for tile in (0, tiles(sms) // 2, tiles(sms) - 1):  # one tile: four blocks
        i = slice(32 * tile, 32 * tile + 32)
        assert steps(cells[i], dts)[0].tobytes() == got[i].tobytes()
    if math == wr.MATH_PORTABLE:
        want = cells.copy()
        rc, cgs = oracle_port.run_cta32(want, perturb=True, max_steps=3)
        assert rc == wr.SUCCESS and cgs == 3
        assert got.tobytes() == want.tobytes()


def test_cta32_clusters_run_at_once(wr, gpu, sms):
    """As long as there are two SMs per tile, a step of like tiles is one wave: a tile takes
    1.4 times as long on two SMs as on four (measured), twice as long in two waves."""
    def step(tiles):
        cells = wr.make_grid(1).repeat(32 * tiles)
        best = np.inf
        with wr.Context(len(cells), 0, wr.MATH_PORTABLE) as ctx:
            for _ in range(4):
                ctx.set_policy(wr.POLICY_GRIDWIDE_INDEPENDENT)
                ctx.upload(cells)
                rc, dt = ctx.prepare(0, 0.0, 0, False)
                assert rc == wr.SUCCESS
                ctx.set_policy(wr.POLICY_GRIDWIDE_CTA32)
                t = time.perf_counter()
                rc, moved = ctx.advance(0, dt, dt)
                best = min(best, time.perf_counter() - t)
                assert rc == wr.SUCCESS and moved == len(cells)
        return best

    few = step(4)
    for tiles in (sms // 4 - 1, sms // 4, sms // 2):
        assert step(tiles) <= 1.7 * few, tiles


@pytest.mark.parametrize("cells_of", [lambda sms: 1, lambda sms: 16 * sms, lambda sms: 16 * sms + 1,
                                      lambda sms: 4095, lambda sms: 4096],
                         ids=["1", "last_32_lanes", "first_16_lanes", "4095", "4096"])
def test_noalloc_shapes(wr, gpu, sms, cells_of):
    """wr_advance_cells_noalloc at 32 and at 16 lanes per cell against the lane-per-cell
    advance of a context."""
    import torch
    n = cells_of(sms)
    cells = wr.make_batch_grid(2, n)
    f = wr.lib().wr_advance_cells_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double,
                  ctypes.POINTER(ctypes.c_int)]
    with wr.Context(n, 0, wr.MATH_PORTABLE) as ctx:
        ctx.set_variant(2)
        ctx.upload(cells)
        rc, dt = ctx.prepare(0, 0.0, 0, True)
        assert rc == wr.SUCCESS
        rc, moved = ctx.advance(0, dt, dt)
        assert rc == wr.SUCCESS
        want = np.empty_like(cells)
        ctx.download(want)
    records = torch.from_numpy(cells.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    count = ctypes.c_int(-1)
    assert f(records.data_ptr(), n, 0, dt, dt, ctypes.byref(count)) == wr.SUCCESS
    assert count.value == moved == n
    assert records.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("grid,variant", [(4, 6), (8, 6), (8, 7)])
def test_lanes_per_cell_equal_reference_cuda_kernel(wr, gpu, grid, variant):
    """The 16-lane advance, which every grid above 16 cells per SM uses, and the 32-lane
    one, each chosen by number, against the reference's own CUDA kernels' final states."""
    want = np.fromfile(os.path.join(GOLDEN, f"refcuda_grid{grid}.bin"), wr.PACKED_FINAL_STATE)
    cells = wr.make_grid(grid)
    with wr.Context(len(cells), 0, wr.MATH_CUDA) as ctx:
        ctx.set_variant(variant)
        ctx.upload(cells)
        rc, _ = ctx.run(True)
        ctx.download(cells)
    assert rc == wr.SUCCESS
    assert wr.pack_final_states(cells, grid).tobytes() == want.tobytes()
