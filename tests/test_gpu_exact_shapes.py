"""The exact replay's transient kernel at the edges of its tiles and chunks,
bit for bit against the oracle (which restates the reference's doubles):
grids narrower than a tile, edges longer than the package CTA's chunk,
per-cell coefficients, and states whose quotients leave the range of the
reciprocal division (the cell then divides plainly)."""
import numpy as np
import pytest

from hotspot_b200 import model as hm
from hotspot_b200 import workloads as W
from oracle.restatement import OracleModel

pytestmark = pytest.mark.gpu


def _pair(sc):
    m, o = hm.from_scenario(sc), OracleModel(sc)
    return m, o, m.vector(o.init_temp), o.vector(o.init_temp)


@pytest.mark.parametrize("rows,cols", [(1, 8), (8, 1), (2, 2), (4, 256), (256, 4), (16, 32), (32, 128)])
def test_transient_shapes_bit_exact(workdir, rows, cols):
    # one block: a cell shared by two blocks is mapped with occupancies that
    # the library's and the oracle's set-up round differently in the last place
    sc = W.scenario_chip2d(workdir, seed=rows + cols, grid=16, steps=3, n_blocks=1)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    m, o, t, to = _pair(sc)
    for k in range(sc.steps):
        p = m.power_vector(sc.block_power[k])
        m.compute_temp(p.copy(), t if k == 0 else None, sc.dt)
        steps = o.compute_temp(p.copy(), to if k == 0 else None, sc.dt)
        assert m.stats()["rk4_steps"] == steps
    assert np.array_equal(t, to) and np.array_equal(m.grid("trans"), o.grid("trans"))
    m.close()


@pytest.mark.parametrize("field", [False, True])
def test_states_outside_the_division_range(workdir, field):
    """Temperatures of zero, 1e-300 K and 1e280 K: the doubles plain division gives."""
    sc = W.scenario_chip2d(workdir, seed=4, grid=16, steps=1, n_blocks=1)
    sc.detailed_3D = field
    m, o, t, to = _pair(sc)
    p = m.power_vector(sc.block_power[0])
    m.compute_temp(p.copy(), t, sc.dt)
    y = m.grid("trans")
    tiny, huge = y.copy(), y.copy()
    tiny[:] = 0.0
    tiny[5:300:7] = 1e-300
    huge[17] = 1e280
    for state in (tiny, huge):
        m.set_grid("trans", state)
        o._y = state.copy()
        o._last_temp = to
        m.compute_temp(p.copy(), None, 1.5e-7)
        o.compute_temp(p.copy(), None, 1.5e-7)
        assert np.array_equal(m.grid("trans"), o.grid("trans"), equal_nan=True)
    m.close()


@pytest.mark.parametrize("rows,cols", [(1, 8), (8, 1), (2, 16), (16, 2), (16, 16), (8, 32)])
def test_steady_shapes_bit_exact(workdir, rows, cols):
    """The wavefront sweeps: lines along either direction, single lines and
    single cells, on every level of the nested iteration."""
    sc = W.scenario_chip2d(workdir, seed=3 * rows + cols, grid=16, steps=1, n_blocks=1)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    m, o, s, so = _pair(sc)
    p = m.power_vector(sc.block_power[0])
    m.steady(p.copy(), s)
    sweeps = o.steady(p.copy(), so)
    assert m.stats()["sweeps"] == sweeps
    assert np.array_equal(s, so) and np.array_equal(m.grid("steady"), o.grid("steady"))
    m.close()
