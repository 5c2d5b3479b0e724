"""What the exact replay's transient kernel is given and takes: per-cell arrays
that a grid has no use for, and device memory."""
import ctypes as C

import numpy as np
import pytest

from hotspot_b200 import FORM_PARITY, _abi
from hotspot_b200 import model as hm
from hotspot_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _device_model(m, rows, cols, cells):
    """A device model with the layers and package of m and one block over the top
    layer; cells: None, or the seven per-cell arrays (None entries allowed)."""
    L, g, nl = _abi.lib(), m.ptr.contents, m.n_layers
    per = [np.array([getattr(g.layers[n], k) for n in range(nl)]) for k in ("rx", "ry", "rz", "c")]
    pack = np.frombuffer(g.pack, dtype=np.float64).copy()
    d = _abi.GridDesc(nl, rows, cols, 12, nl - 2, nl - 1, -1, -1, -1, int(cells is not None), 0, 1, m.config.ambient,
                      g.width, g.height, 0.0, *[_abi.dptr(a) for a in per], _abi.dptr(pack))
    dev = C.c_void_p()
    assert L.hsb_dev_create(C.byref(dev), C.byref(d)) == 0, L.hsb_dev_last_error()
    if cells is not None:
        assert L.hsb_dev_set_cells(dev, *[None if a is None else _abi.dptr(a) for a in cells]) == 0
    plane, n = rows * cols, nl * rows * cols
    ptr = np.minimum(np.arange(n + 1), plane).astype(np.int32)
    blk, one = np.zeros(plane, np.int32), np.ones(plane)
    g2b = np.array([0, 0, rows, 0, cols], np.int32)
    area = g.width * g.height
    ints = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))
    assert L.hsb_dev_set_maps(dev, ints(ptr), ints(blk), _abi.dptr(one), _abi.dptr(one * area), area / plane, ints(g2b)) == 0
    return dev


def _interval(dev, n, ambient):
    L = _abi.lib()
    y, p, out = np.full(n + 12, ambient), np.zeros(13), np.zeros(13)
    p[0] = 20.0
    st, opts = _abi.Stats(), _abi.SolverOpts(FORM_PARITY, 0, 0.0, 0)
    assert L.hsb_dev_set_state(dev, 0, _abi.dptr(y)) == 0
    rc = L.hsb_dev_transient(dev, _abi.dptr(p), None, 1e-5, _abi.dptr(out), C.byref(opts), C.byref(st))
    assert L.hsb_dev_get_state(dev, 0, _abi.dptr(y)) == 0
    return rc, y


@pytest.mark.parametrize("rows,cols", [(1, 8), (8, 1), (8, 8)])
def test_cells_without_the_arrays_they_do_not_need(workdir, rows, cols):
    """A grid of one row (column) has no resistances to the north and south (east
    and west), and its owner need not pass arrays of them: the doubles of the
    same model with per-layer coefficients.  Without those it does need the call
    is refused."""
    sc = W.scenario_chip2d(workdir, seed=3, grid=16, steps=1, n_blocks=1)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    m = hm.from_scenario(sc)
    g, nl = m.ptr.contents, m.n_layers
    per_cell = lambda v: np.repeat(np.asarray(v, dtype=np.float64), rows * cols)
    layer = [g.layers[n] for n in range(nl)]
    ns = per_cell([l.rx / 2.0 + l.rx / 2.0 for l in layer])
    ew = per_cell([l.ry / 2.0 + l.ry / 2.0 for l in layer])
    above = per_cell([0.0] + [l.rz for l in layer[:-1]])
    below = per_cell([l.rz for l in layer])
    cells = [None if rows == 1 else ns, None if rows == 1 else ns, None if cols == 1 else ew,
             None if cols == 1 else ew, above, below, per_cell([l.c for l in layer])]
    L, states = _abi.lib(), []
    for a in (None, cells):
        dev = _device_model(m, rows, cols, a)
        rc, y = _interval(dev, m.n_cells, m.config.ambient)
        assert rc == 0, L.hsb_dev_last_error()
        states.append(y)
        L.hsb_dev_destroy(dev)
    assert np.max(states[0]) > m.config.ambient and np.array_equal(*states)
    for k in (5, 6):
        dev = _device_model(m, rows, cols, cells[:k] + [None] + cells[k + 1:])
        rc, _ = _interval(dev, m.n_cells, m.config.ambient)
        assert rc != 0 and b"lack" in L.hsb_dev_last_error()
        L.hsb_dev_destroy(dev)
    m.close()


@pytest.mark.parametrize("detailed", [False, True])
def test_work_vectors_and_short_memory(workdir, detailed):
    """A step keeps six vectors beside the model's four (and the reciprocals of
    per-cell coefficients).  Where memory is short it does with five and without
    the reciprocals, no more than the launch per stage kept, and gives the same
    bits: two intervals with rejected attempts."""
    import torch

    sc = W.scenario_chip2d(workdir, seed=8, grid=512, steps=1, n_blocks=4)
    sc.detailed_3D = detailed

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    def run(room):
        m = hm.from_scenario(sc)
        before = free()
        hog = torch.empty(before - room, dtype=torch.uint8, device="cuda") if room else None
        p, t = m.power_vector(sc.block_power[0]), m.vector(m.config.init_temp)
        m.compute_temp(p.copy(), t, 1e-5)
        del hog
        used = before - free()
        m.compute_temp(p.copy(), None, 2e-3)
        st, y = m.stats(), m.grid("trans")
        m.close()
        return used, st, y

    vec = 8 * 4 * 512 * 512
    run(0)                    # loads the kernels
    used, st, y = run(0)
    assert st["rk4_attempts"] > st["rk4_steps"]
    assert used <= (6.5 + 7 * detailed) * vec
    short, sts, ys = run(int(5.6 * vec))
    assert short <= 5.6 * vec
    assert (st["rk4_steps"], st["rk4_attempts"], st["slope_evals"]) == (sts["rk4_steps"], sts["rk4_attempts"], sts["slope_evals"])
    assert np.array_equal(y, ys)
