"""The multifrontal linear solve (schedule 4) against the level launches (schedule 0) on the same batches: the host plan on
every ordering (CPU), the kernels at the edges of their lane pairs, 64-lane warps and CTA shapes (GPU)."""
import numpy as np
import pytest

from conftest import grid

_SMALL = {}


def grid600():
    """The smallest size class that takes the multifrontal solve."""
    if not _SMALL:
        from olfgpu import packing, synthetic
        g = synthetic.calibrate(synthetic.generate(synthetic.GridSpec("grid600", 600, 960, 120, 390, 0.10, seed=600)))
        _SMALL["g"] = (g, packing.pack(g))
    return _SMALL["g"]


@pytest.mark.parametrize("name", ["grid118", "grid300", "grid2000"])
@pytest.mark.parametrize("ordering", [0, 1, 2, 3, 16, 19])
def test_plan_holds(engine_lib, name, ordering):
    """Every LU block stored once, every Jacobian block and update block added once at its place, no update matrix
    overwritten before its parent has read it (the check is olfgpu_structure_check_plan's)."""
    from olfgpu import native
    if ordering == 2 and name != "grid118":
        pytest.skip("the natural order fills the larger grids")
    _, p = grid(name)
    violations, first = native.Structure(p, ordering).check_plan()
    assert violations == 0, first


@pytest.mark.parametrize("name,ordering,blocks", [
    ("grid300", 19, 0), ("grid600", 19, None), ("grid600", 2, 0), ("grid2000", 19, 8356), ("grid2000", 1, 0),
    ("grid2000", 8, 0), ("grid9241", 19, 41424), ("grid9241", 0, 36715), ("grid9241", 1, 0), ("grid13659", 0, 0)])
def test_which_structures_have_a_plan(engine_lib, name, ordering, blocks):
    """No plan for a small grid, a deferred-L plan and an order with more than 40 rows below some pivot: 104 in the natural
    order of 600 buses, 52 and 128 by nested dissection, 44 by minimum degree on 13,659.  The update matrices' blocks a
    lane are the memory a context takes."""
    from olfgpu import native
    p = (grid600() if name == "grid600" else grid(name))[1]
    s = native.Structure(p, ordering)
    mf = s.multifrontal()
    assert (mf["nodes"] > 0) == (blocks != 0)
    assert blocks is None or mf["update_blocks"] == blocks
    assert mf["rows_below"] <= 40 and mf["front_rows"] <= 41
    assert s.check_plan()[0] == 0


# Both schedules solve the same 2x2 block systems in another summation order: a step's relative difference is about
# eps * cond(J), 2e-16 * 1e5, and the iterations contract it; 1e-10 leaves a factor of five.
STATE_TOL = 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("name,ordering,count", [
    ("grid600", 19, 1), ("grid600", 0, 2), ("grid600", 1, 3), ("grid600", 2, 5), ("grid600", 16, 33), ("grid600", 3, 65),
    ("grid2000", 19, 1), ("grid2000", 19, 17), ("grid2000", 16, 64), ("grid2000", 0, 97)])
def test_states_match_the_level_launches(engine_lib, name, ordering, count):
    """Odd and even lane counts, one and several lane groups, every ordering (the natural one has the widest fronts)."""
    from olfgpu import native, synthetic
    g, p = grid600() if name == "grid600" else grid(name)
    outs = synthetic.draw_outages(g, count, seed=7 + count)
    dis = p.outage_masks(outs)
    s = native.Structure(p, ordering)
    res = []
    for schedule in ((0, 0, 256), (4, 0, 256)):
        ctx = native.BatchContext(s, count)
        ctx.set_schedule(*schedule)
        res.append(ctx.solve(p.x_base, p.target, p.base_row_mode, dis))
    a, b = res
    conv = a[:, -1] == 0
    assert np.array_equal(a[:, -1], b[:, -1]) and np.array_equal(a[conv, p.n], b[conv, p.n])
    assert conv.any() and np.max(np.abs(a[conv, :p.n] - b[conv, :p.n])) < STATE_TOL


@pytest.mark.gpu
def test_a_lane_does_not_depend_on_its_batch(engine_lib):
    """Lane pairs, CTA shapes and strands follow the batch size; every sum keeps its order: the same bits."""
    from olfgpu import native, synthetic
    g, p = grid("grid2000")
    outs = synthetic.draw_outages(g, 150, seed=5)
    s = native.Structure(p, native.PLAN_DEFAULT)
    rows = {}
    for count in (1, 2, 9, 40, 150):
        ctx = native.BatchContext(s, count)
        ctx.set_schedule(native.LEVELS_SHARED_ALL, 0, 256)
        rows[count] = ctx.solve(p.x_base, p.target, p.base_row_mode, p.outage_masks(outs[:count]))[0].copy()
    for count, row in rows.items():
        assert np.array_equal(row, rows[150]), count
