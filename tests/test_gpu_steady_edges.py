"""The fast steady solvers where their iterations have nothing to do, are given
something they cannot solve, or meet a model that has changed."""
import numpy as np
import pytest

from hotspot_b200 import FORM_FAST, STEADY_AUTO, STEADY_BICGSTAB, _abi
from hotspot_b200 import model as hm
from hotspot_b200 import workloads as W
from hotspot_b200._abi import HotspotError

pytestmark = pytest.mark.gpu

# one level; whole passes in the cluster; tiles above it; kernel by kernel
MG_CASES = [(4, 8, False), (16, 16, False), (256, 128, False), (16, 16, True)]


def _chip(workdir, rows, cols, detailed, seed=5):
    sc = W.scenario_chip2d(workdir, seed=seed, grid=16, steps=1, n_blocks=3)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    sc.detailed_3D = detailed
    return sc


@pytest.mark.parametrize("rows,cols,detailed", MG_CASES)
def test_mg_steady_without_power(workdir, rows, cols, detailed):
    """No power: everything is at ambient, where the first residual is zero to
    the last bit, and the step lengths of the conjugate gradients are 0 / 0."""
    m = hm.from_scenario(_chip(workdir, rows, cols, detailed))
    m.set_solver(FORM_FAST)
    s = m.vector()
    for _ in range(2):
        m.steady(m.vector(), s)
        assert np.array_equal(m.grid("steady"), np.full(m.n_cells + m.n_extra, m.config.ambient))
        assert np.array_equal(s, m.vector(m.config.ambient))
    m.close()


def _uchan(workdir, seed=2, **kw):
    return W.scenario_microchannel(workdir, seed=seed, **(kw or dict(
        grid=32, die=2e-3, channel_w=125e-6, channel_h=125e-6, pitch=250e-6, blocks=8)))


def _power_that_is_no_number(sc):
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST)
    p = m.power_vector(sc.block_power[0])
    s, t = m.vector(), m.vector()
    m.steady(p.copy(), s)
    bad = p.copy()
    bad[np.flatnonzero(p)[0]] = np.nan
    with pytest.raises(HotspotError, match="not finite"):
        m.steady(bad, t)
    m.steady(p.copy(), t)
    assert np.array_equal(s, t)
    m.close()


@pytest.mark.parametrize("rows,cols,detailed", MG_CASES)
def test_mg_steady_of_a_power_that_is_no_number(workdir, rows, cols, detailed):
    """An error, not temperatures that are no numbers; the model solves on."""
    _power_that_is_no_number(_chip(workdir, rows, cols, detailed))


def test_bicgstab_steady_of_a_power_that_is_no_number(workdir):
    _power_that_is_no_number(_uchan(workdir))


@pytest.mark.parametrize("what,method", [("chip", STEADY_AUTO), ("chip", STEADY_BICGSTAB), ("uchan", STEADY_AUTO)])
def test_steady_after_the_package_changed(workdir, what, method):
    """A model that has solved once and is given another spreader and sink (the
    package's and the edges' conductances change) solves as a fresh model with
    them does: the same passes and the same bits."""
    sc = _uchan(workdir) if what == "uchan" else _chip(workdir, 32, 32, False)
    new = {"s_spreader": "0.05", "s_sink": "0.09"}
    m = hm.from_scenario(sc)
    sc.config.update(new)
    f = hm.from_scenario(sc)
    p, s, t = m.power_vector(sc.block_power[0]), m.vector(), m.vector()
    for x in (m, f):
        x.set_solver(FORM_FAST, method)
    m.steady(p.copy(), s)
    cfg = m.ptr.contents.config
    cfg.s_spreader, cfg.s_sink = float(new["s_spreader"]), float(new["s_sink"])
    hm.populate_R_model(m, m._flp)
    m.steady(p.copy(), s)
    f.steady(p.copy(), t)
    a, b = m.stats(), f.stats()
    assert (a["refinements"], a["cycles"]) == (b["refinements"], b["cycles"])
    assert np.array_equal(m.grid("steady"), f.grid("steady")) and np.array_equal(s, t)
    m.close()
    f.close()


@pytest.mark.parametrize("rows,cols,tol", [(4, 16, 1e-9), (1, 16, 1e-9), (4, 8, 1e-10), (8, 4, 1e-10)])
def test_mg_single_level_refinements(workdir, rows, cols, tol):
    """Grids that are one level of the multigrid: its exact solve takes the
    residual of each iteration, package nodes included, so a per-layer model
    (whole passes in the cluster) needs no more passes than the same model with
    per-cell coefficients (kernel by kernel)."""
    passes = []
    for detailed in (False, True):
        sc = _chip(workdir, rows, cols, detailed)
        m = hm.from_scenario(sc)
        m.set_solver(FORM_FAST, steady_tol=tol)
        m.steady(m.power_vector(sc.block_power[0]), m.vector())
        passes.append(m.stats()["refinements"])
        m.close()
    assert passes[0] <= passes[1]


def test_mg_out_of_memory_then_again(workdir):
    """A steady solve that runs out of device memory while it sets its workspace
    up (the last of its vectors does not fit) reports that, and the model solves
    once there is room; nothing stays allocated."""
    import torch

    sc = _chip(workdir, 1024, 1024, False)

    def model():
        m = hm.from_scenario(sc)
        m.set_solver(FORM_FAST)
        return m, m.power_vector(sc.block_power[0])

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    for _ in range(2):        # the first loads the kernels, the second is measured
        m, p = model()
        want = m.vector()
        before = free()
        m.steady(p.copy(), want)
        workspace = before - free()
        m.close()
    vec = 4 * 4 * 1024 * 1024
    assert workspace > 10 * vec
    raised, base = 0, free()
    for short in (4 << 20, vec // 2, vec, 6 * vec):
        m, p = model()
        hog = torch.empty(free() - (workspace - short), dtype=torch.uint8, device="cuda")
        try:
            m.steady(p.copy(), m.vector())
        except HotspotError as e:
            assert "memory" in str(e)
            raised += 1
        del hog
        free()
        s = m.vector()
        m.steady(p.copy(), s)
        assert np.array_equal(s, want)
        m.close()
        assert free() > base - vec
    assert raised >= 2


@pytest.mark.parametrize("rows,cols", [(4, 8), (32, 32), (256, 128)])
def test_mg_after_an_operator_without_inverse(workdir, rows, cols):
    """A model that has solved, then gets conductances of zero throughout (its
    coarsest operator has no inverse any more): the solve reports that it cannot,
    and with the conductances back it gives the same bits."""
    sc = _chip(workdir, rows, cols, False)
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST)
    p, s, t = m.power_vector(sc.block_power[0]), m.vector(), m.vector()
    m.steady(p.copy(), s)
    inf = np.full(52, np.inf)
    L = _abi.lib()
    assert L.hsb_dev_set_layers(L.hsb_grid_device(m.ptr), *[_abi.dptr(inf)] * 5, m.config.ambient, 0.016, 0.016, 0.0) == 0
    with pytest.raises(HotspotError):
        m.steady(p.copy(), t)
    hm.populate_R_model(m, m._flp)
    hm.populate_C_model(m, m._flp)
    m.steady(p.copy(), t)
    assert np.array_equal(s, t)
    m.close()


@pytest.mark.parametrize("rows,cols", [(8, 1), (64, 1), (1, 8), (1, 1)])
def test_bicgstab_steady_of_a_single_column(workdir, rows, cols):
    """A grid of one column has no planes of the second colour; the plane solver
    gives what the multigrid solver gives.  Both stop with corrections of 1e-7 K
    at most, and contract by more than ten."""
    sc = _chip(workdir, rows, cols, False)
    m, g = hm.from_scenario(sc), hm.from_scenario(sc)
    m.set_solver(FORM_FAST, STEADY_BICGSTAB)
    g.set_solver(FORM_FAST)
    p, s, t = m.power_vector(sc.block_power[0]), m.vector(), m.vector()
    for _ in range(2):
        m.steady(p.copy(), s)
    g.steady(p.copy(), t)
    assert np.max(t) > m.config.ambient + 1.0
    assert np.max(np.abs(s - t)) < 1e-6
    m.close()
    g.close()


def test_bicgstab_steady_of_many_passes(workdir):
    """A grid of 128 times more rows than columns, among the slowest to converge:
    solved within the default number of passes.  Bar: the fast form's (0.01 K)."""
    from oracle.restatement import OracleModel

    sc = W.scenario_chip2d(workdir, seed=3588, grid=16, steps=1, n_blocks=5)
    sc.config.update(grid_rows="512", grid_cols="4")
    m, o = hm.from_scenario(sc), OracleModel(sc)
    m.set_solver(FORM_FAST, STEADY_BICGSTAB)
    p = m.power_vector(sc.block_power[0])
    m.steady(p.copy(), m.vector())
    assert np.max(np.abs(m.grid("steady") - o.steady_direct(p)[0])) <= 0.01
    m.close()


@pytest.mark.parametrize("detailed", [False, True])
@pytest.mark.parametrize("rows,cols,chip_layers", [(17, 31, 1), (33, 48, 2), (100, 100, 1), (300, 200, 1), (300, 300, 1),
                                                   (8, 2, 5), (300, 200, 8)])
def test_mg_kernel_by_kernel_vectors(workdir, rows, cols, chip_layers, detailed):
    """The kernel-by-kernel form, on grids where a level's vector and its package
    slots end at the end of the memory they are given (the coarsest level too
    large for a dense inverse, or per-cell coefficients): every solve of a model
    gives the same bits, with the layers' resistances and with the same ones cell
    by cell, and is a solution by its FP64 residual (33x48 is a single level that
    the smoother alone does not solve within the default passes: the bits of where
    it gives up)."""
    import ctypes as C

    from test_gpu_exact_workspace import _device_model

    m = hm.from_scenario(W.scenario_random_chip(workdir, np.random.default_rng(2), "x", side=32, chip_layers=chip_layers,
                                                steps=1))
    L, layer, nl = _abi.lib(), [m.ptr.contents.layers[n] for n in range(m.n_layers)], m.n_layers
    per_cell = lambda v: np.repeat(np.asarray(v, dtype=np.float64), rows * cols)
    ns, ew = per_cell([l.rx for l in layer]), per_cell([l.ry for l in layer])
    cells = [ns, ns, ew, ew, per_cell([0.0] + [l.rz for l in layer[:-1]]), per_cell([l.rz for l in layer]),
             per_cell([l.c for l in layer])]
    p, out = np.zeros(13), np.zeros(13)
    p[0] = 20.0
    states = []
    for a in ((cells,) if detailed or rows * cols == 16 else (None, cells)):   # (8x2 per layer runs in the cluster)
        dev = _device_model(m, rows, cols, a)
        for _ in range(2):
            st, opts = _abi.Stats(), _abi.SolverOpts(FORM_FAST, STEADY_AUTO, 0.0, 0)
            rc = L.hsb_dev_steady(dev, _abi.dptr(p), _abi.dptr(out), C.byref(opts), C.byref(st))
            assert rc == 0 or (rows == 33 and b"did not converge" in L.hsb_dev_last_error()), L.hsb_dev_last_error()
            y = np.zeros(nl * rows * cols + 12)
            assert L.hsb_dev_get_state(dev, 1, _abi.dptr(y)) == 0
            assert rc or st.residual < 1e-5
            assert np.min(y) > m.config.ambient
            states.append(y)
        L.hsb_dev_destroy(dev)
    for y in states[1:]:
        assert np.array_equal(y, states[0])
    m.close()


@pytest.mark.parametrize("detailed", [False, True])
@pytest.mark.parametrize("rows,cols,chip_layers", [(1, 1, 1), (2, 2, 1), (4, 4, 1), (4, 8, 1), (2, 2, 4), (32, 32, 4)])
def test_mg_steady_of_next_to_no_power(workdir, rows, cols, chip_layers, detailed):
    """Residuals that the iteration brings to the end of FP32's range: powers of
    1e-20 W and less heat by less than a temperature's last place, so everything
    is at ambient to the bit."""
    import ctypes as C

    from test_gpu_exact_workspace import _device_model

    m = hm.from_scenario(W.scenario_random_chip(workdir, np.random.default_rng(32), "x", side=32, chip_layers=chip_layers,
                                                steps=1))
    L, layer, nl = _abi.lib(), [m.ptr.contents.layers[n] for n in range(m.n_layers)], m.n_layers
    per_cell = lambda v: np.repeat(np.asarray(v, dtype=np.float64), rows * cols)
    ns, ew = per_cell([l.rx for l in layer]), per_cell([l.ry for l in layer])
    cells = [ns, ns, ew, ew, per_cell([0.0] + [l.rz for l in layer[:-1]]), per_cell([l.rz for l in layer]),
             per_cell([l.c for l in layer])]
    dev = _device_model(m, rows, cols, cells if detailed else None)
    p, out, y = np.zeros(13), np.zeros(13), np.zeros(nl * rows * cols + 12)
    for power in (1e-20, 1e-25, 1e-30, 1e-35, 1e-38, 1e-44, 1e-300):
        p[0] = power
        st, opts = _abi.Stats(), _abi.SolverOpts(FORM_FAST, STEADY_AUTO, 0.0, 0)
        rc = L.hsb_dev_steady(dev, _abi.dptr(p), _abi.dptr(out), C.byref(opts), C.byref(st))
        assert rc == 0, (power, L.hsb_dev_last_error())
        assert L.hsb_dev_get_state(dev, 1, _abi.dptr(y)) == 0
        assert np.array_equal(y, np.full(y.size, m.config.ambient)), power
    L.hsb_dev_destroy(dev)
    m.close()
