"""The fast forms (HSB_FORM_FAST) against the FP64 oracle.

Transient: FP32 stencil stages with FP64 state, error norm and step control
on the device; compared with the oracle's exact FP64 replay of the
reference (same adaptive algorithm), bar max |dT| <= 0.01 K.
Steady: FP32 multigrid-preconditioned CG inside FP64 iterative refinement;
compared with the converged FP64 solution of the same system by sparse
direct LU, bar max |dT| <= 0.01 K (the solver converges far below it).
"""
import glob
import os

import numpy as np
import pytest

from hotspot_b200 import FORM_FAST, FORM_FAST_PASSES
from hotspot_b200 import model as hm
from hotspot_b200 import workloads as W
from oracle.restatement import OracleModel

pytestmark = pytest.mark.gpu
TOL = 0.01


def _transient(sc, steps):
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST)
    o = OracleModel(sc)
    t, to = m.vector(o.init_temp), o.vector(o.init_temp)
    worst = 0.0
    for k in range(steps):
        p = m.power_vector(sc.block_power[k])
        m.compute_temp(p.copy(), t if k == 0 else None, sc.dt)
        o.compute_temp(p.copy(), to if k == 0 else None, sc.dt)
        worst = max(worst, float(np.max(np.abs(t - to))))
    grid_err = float(np.max(np.abs(m.grid("trans") - o.grid("trans"))))
    m.close()
    return worst, grid_err


@pytest.mark.parametrize("grid", [32, 64])
def test_fast_transient_chip2d(workdir, grid):
    sc = W.scenario_chip2d(workdir, seed=11, grid=grid, steps=40)
    worst, grid_err = _transient(sc, sc.steps)
    assert worst <= TOL and grid_err <= TOL


def test_fast_transient_stack(workdir):
    sc = W.scenario_stack3d(workdir, seed=12, grid=64, steps=20, n_blocks=16)
    worst, grid_err = _transient(sc, sc.steps)
    assert worst <= TOL and grid_err <= TOL


def test_fast_transient_detailed(workdir):
    sc = W.scenario_stack3d(workdir, seed=13, grid=32, steps=10, n_blocks=10)
    sc.detailed_3D = True
    worst, grid_err = _transient(sc, sc.steps)
    assert worst <= TOL and grid_err <= TOL


def test_fast_transient_microchannel(workdir):
    sc = W.scenario_microchannel(workdir, seed=2, grid=32, die=2e-3, channel_w=125e-6,
                                 channel_h=125e-6, pitch=250e-6, blocks=8)
    sc.block_power = np.repeat(sc.block_power, 3, axis=0)
    sc.dt = 1e-5
    worst, grid_err = _transient(sc, 3)
    assert worst <= TOL and grid_err <= TOL


@pytest.mark.parametrize("builder,grid", [("chip2d", 64), ("stack3d", 64), ("detailed", 32)])
def test_mg_steady_converged(workdir, builder, grid):
    if builder == "chip2d":
        sc = W.scenario_chip2d(workdir, seed=21, grid=grid, steps=2)
    else:
        sc = W.scenario_stack3d(workdir, seed=22, grid=grid, steps=2, n_blocks=14)
        sc.detailed_3D = builder == "detailed"
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST)
    o = OracleModel(sc)
    avg = m.power_vector(sc.block_power.mean(0))
    s = m.vector()
    m.steady(avg.copy(), s)
    T, Tb = o.steady_direct(avg)
    assert np.max(np.abs(s - Tb)) <= TOL
    assert np.max(np.abs(m.grid("steady") - T)) <= TOL
    st = m.stats()
    assert st["refinements"] >= 1
    m.close()


@pytest.mark.parametrize("builder", ["chip2d", "stack3d", "detailed"])
def test_krylov_form_matches_stage_form(workdir, builder):
    """The default fast transient (step-doubling RK4 evaluated through Krylov
    vectors of the affine slope operator) against the same fast arithmetic
    evaluated stage by stage: same accepted steps, temperatures within 1e-3 K."""
    from hotspot_b200 import FORM_FAST_STAGES
    if builder == "chip2d":
        sc = W.scenario_chip2d(workdir, seed=31, grid=64, steps=25)
    else:
        sc = W.scenario_stack3d(workdir, seed=32, grid=64, steps=25, n_blocks=12)
        sc.detailed_3D = builder == "detailed"
    runs = []
    for form in (FORM_FAST, FORM_FAST_STAGES):
        m = hm.from_scenario(sc)
        m.set_solver(form)
        t = m.vector(m.config.init_temp)
        out = []
        tot = {"rk4_steps": 0, "rk4_attempts": 0, "fallbacks": 0}
        for k in range(sc.steps):
            m.compute_temp(m.power_vector(sc.block_power[k]), t if k == 0 else None, sc.dt)
            out.append(t.copy())
            st = m.stats()
            for key in tot:
                tot[key] += st[key]
        runs.append((np.array(out), m.grid("trans"), tot))
        m.close()
    (a, ga, sa), (b, gb, sb) = runs
    assert sa["rk4_steps"] == sb["rk4_steps"] and sa["rk4_attempts"] == sb["rk4_attempts"]
    assert sa["fallbacks"] == 0
    assert np.max(np.abs(a - b)) <= 1e-3 and np.max(np.abs(ga - gb)) <= 1e-3


@pytest.mark.parametrize("grid,seed", [(32, 41), (64, 42)])
def test_bicgstab_microchannel_steady(workdir, grid, seed):
    """The non-symmetric steady system of a microchannel model (advection
    terms +-Cv*flow/2, which the reference can only hand to SuperLU) by FP32
    BiCGStab with FP64 refinement, against FP64 sparse LU of the same
    system: bar max |dT| <= 0.01 K."""
    from hotspot_b200 import STEADY_BICGSTAB
    sc = W.scenario_microchannel(workdir, seed=seed, grid=grid, die=grid * 20e-6, blocks=8)
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST, STEADY_BICGSTAB)
    o = OracleModel(sc)
    p = m.power_vector(sc.block_power[0])
    s = m.vector()
    m.steady(p.copy(), s)
    T, Tb = o.steady_direct(p)
    st = m.stats()
    err_b = float(np.max(np.abs(s - Tb)))
    err_g = float(np.max(np.abs(m.grid("steady") - T)))
    m.close()
    assert err_b <= TOL and err_g <= TOL, (err_b, err_g, st)
    assert st["refinements"] >= 1 and st["residual"] < 1e-6


def test_bicgstab_symmetric_model(workdir):
    """The same solver on a model without advection agrees with the direct solve."""
    from hotspot_b200 import STEADY_BICGSTAB
    sc = W.scenario_stack3d(workdir, seed=43, grid=64, steps=2, n_blocks=10)
    sc.detailed_3D = True
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST, STEADY_BICGSTAB)
    o = OracleModel(sc)
    avg = m.power_vector(sc.block_power.mean(0))
    s = m.vector()
    m.steady(avg.copy(), s)
    T, Tb = o.steady_direct(avg)
    err = float(np.max(np.abs(m.grid("steady") - T)))
    m.close()
    assert np.max(np.abs(s - Tb)) <= TOL and err <= TOL, err


@pytest.mark.parametrize("builder", ["chip2d", "stack3d", "detailed"])
def test_trace_equals_single_intervals(workdir, builder):
    """K intervals in one persistent launch (hsb_dev_transient_trace) give the
    results of K single-interval calls of the fast form, bit for bit."""
    if builder == "chip2d":
        sc = W.scenario_chip2d(workdir, seed=51, grid=64, steps=12)
    else:
        sc = W.scenario_stack3d(workdir, seed=52, grid=64, steps=12, n_blocks=12)
        sc.detailed_3D = builder == "detailed"
    a, b = hm.from_scenario(sc), hm.from_scenario(sc)
    a.set_solver(FORM_FAST)
    t = a.vector(a.config.init_temp)
    powers = np.stack([a.power_vector(sc.block_power[k]) for k in range(sc.steps)])
    steps_a = 0
    for k in range(sc.steps):
        a.compute_temp(powers[k].copy(), t if k == 0 else None, sc.dt)
        steps_a += a.stats()["rk4_steps"]
    out, st = b.compute_trace(powers, b.vector(b.config.init_temp), sc.dt)
    assert st["rk4_steps"] == steps_a
    assert np.array_equal(out, t)
    assert np.array_equal(a.grid("trans"), b.grid("trans"))
    a.close()
    b.close()


def test_forms_alternate_on_one_model(workdir):
    """Switching one model between the parity and the fast forms from call to
    call: each form keeps its own state buffers and swaps them as steps are
    accepted, so the fast form's replayed interval graphs must follow the
    buffers' current roles.  The trajectory stays within 0.01 K of the FP64
    replay."""
    from hotspot_b200 import FORM_PARITY
    sc = W.scenario_chip2d(workdir, seed=71, grid=32, steps=12)
    m, o = hm.from_scenario(sc), OracleModel(sc)
    t, to = m.vector(o.init_temp), o.vector(o.init_temp)
    forms = [FORM_FAST, FORM_FAST, FORM_PARITY, FORM_FAST, FORM_FAST, FORM_PARITY, FORM_PARITY, FORM_FAST,
             FORM_FAST, FORM_FAST, FORM_PARITY, FORM_FAST]
    for k, form in enumerate(forms):
        m.set_solver(form)
        p = m.power_vector(sc.block_power[k])
        m.compute_temp(p.copy(), t if k == 0 else None, sc.dt)
        o.compute_temp(p.copy(), to if k == 0 else None, sc.dt)
        assert np.max(np.abs(t - to)) <= TOL, k
    assert np.max(np.abs(m.grid("trans") - o.grid("trans"))) <= TOL
    m.close()


def test_mg_steady_secondary_path(workdir):
    """The MG-PCG steady solve on the secondary heat path (substrate, solder
    and PCB layers, 28 package nodes; the steady package equations of
    temperature_grid.c:2228-2379) against the reference's own steady result
    (golden vectors of the reference build, which stops within 1e-3 K of the
    fixed point) and, on a 64x64 chip, against the FP64 replay of the
    reference's Gauss-Seidel: 0.01 K, with a converged FP64 residual."""
    from test_gpu_parity import _golden
    sc, n, g = _golden(workdir, "secondary_16")
    m = hm.from_scenario(sc)
    m.set_solver(FORM_FAST)
    s = m.vector()
    m.steady(g["steady_power"].copy(), s)
    assert np.max(np.abs(s - g["steady"])) <= TOL
    assert np.max(np.abs(m.grid("steady") - g["grid_steady"])) <= TOL
    assert m.stats()["refinements"] >= 1
    m.close()
    sc = W.scenario_chip2d(workdir, seed=23, grid=64, steps=2)
    sc.config["model_secondary"] = "1"
    out = []
    for form in (FORM_FAST, None):
        m = hm.from_scenario(sc)
        if form is not None:
            m.set_solver(form)
        p = m.power_vector(sc.block_power.mean(0))
        s = m.vector()
        m.steady(p.copy(), s)
        out.append((s, m.grid("steady"), m.stats()))
        m.close()
    (sf, gf, stf), (sr, gr, _) = out
    assert np.max(np.abs(sf - sr)) <= TOL and np.max(np.abs(gf - gr)) <= TOL
    assert stf["residual"] < 1e-6


@pytest.mark.parametrize("rows,cols,dt", [(4, 8, 3.333e-6), (8, 4, 3.333e-6), (16, 256, 1e-5), (256, 16, 1e-5), (64, 128, 2e-3),
                                          (128, 64, 3.333e-6)])
def test_paired_passes_shapes(workdir, rows, cols, dt):
    """The paired-pass transient kernel at the edges of its tiles: grids
    smaller than a tile, tiles along one edge only, long intervals with
    rejected attempts, and a trace of intervals in one launch against the
    same intervals one by one.  Bar: the fast form's (0.01 K); the steps are
    those of the same arithmetic one pass at a time (FP32 error norms need not
    take the FP64 steps on long intervals)."""
    sc = W.scenario_stack3d(workdir, seed=rows + cols, grid=16, steps=3, n_blocks=3)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    m, n, q, o = hm.from_scenario(sc), hm.from_scenario(sc), hm.from_scenario(sc), OracleModel(sc)
    m.set_solver(FORM_FAST)
    q.set_solver(FORM_FAST_PASSES)
    t, to, tq = m.vector(o.init_temp), o.vector(o.init_temp), m.vector(o.init_temp)
    ps = np.stack([m.power_vector(sc.block_power[k]) for k in range(sc.steps)])
    for k in range(sc.steps):
        m.compute_temp(ps[k].copy(), t if k == 0 else None, dt)
        q.compute_temp(ps[k].copy(), tq if k == 0 else None, dt)
        o.compute_temp(ps[k].copy(), to if k == 0 else None, dt)
        a, b = m.stats(), q.stats()
        assert (a["rk4_steps"], a["rk4_attempts"], a["slope_evals"]) == (b["rk4_steps"], b["rk4_attempts"], b["slope_evals"])
    assert m.transient_kernel() == "passes"
    assert np.max(np.abs(m.grid("trans") - o.grid("trans"))) <= TOL
    tn, _ = n.compute_trace(ps, n.vector(o.init_temp), dt, form=FORM_FAST)
    assert np.array_equal(n.grid("trans"), m.grid("trans")) and np.array_equal(tn, t)
    for x in (m, n, q):
        x.close()


@pytest.mark.parametrize("rows,cols,kernel", [(4, 8, "rk4_pair_kernel"), (128, 64, "rk4_pair_kernel"),
                                              (1024, 64, "rk4_pair_kernel"), (1024, 128, "rk4_krylov_kernel")])
def test_which_pass_kernel_runs(workdir, rows, cols, kernel):
    """The paired passes take every grid that tiles of 512 columns put on the
    SMs (75776 columns on 148) and no larger one; a model told to go pass by
    pass never takes them."""
    sc = W.scenario_stack3d(workdir, seed=1, grid=16, steps=1, n_blocks=3)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    for form, want in ((FORM_FAST, kernel), (FORM_FAST_PASSES, "rk4_krylov_kernel")):
        m = hm.from_scenario(sc)
        m.set_solver(form)
        assert m.transient_kernel_name() == ""
        m.compute_temp(m.power_vector(sc.block_power[0]), m.vector(m.config.init_temp), sc.dt)
        assert m.transient_kernel_name() == want and m.transient_kernel() == "passes"
        m.close()


def _narrow(workdir, by):
    """Scale the x extents of every floorplan in the directory."""
    for f in glob.glob(os.path.join(workdir, "*.flp")):
        rows = [l.split() for l in open(f) if l.strip() and not l.startswith("#")]
        with open(f, "w") as o:
            for r in rows:
                o.write("%s\t%.9e\t%s\t%.9e\t%s\n" % (r[0], float(r[1]) * by, r[2], float(r[3]) * by, r[4]))


@pytest.mark.parametrize("rows,cols,layers", [(4, 4, 1), (8, 32, 3), (16, 16, 8), (32, 64, 4), (256, 32, 1), (512, 16, 6),
                                              (2048, 8, 6)])
def test_bicgstab_plane_shapes(workdir, rows, cols, layers):
    """The plane solver at the edges of its parts: planes that are one dense
    block, few and many reduction steps, an odd number of layers, factors read
    from global memory (8 layers of 512 rows) and vectors kept there as well
    (2048 rows; on the narrow grids the die is narrowed to cells of 4:1).  Against the FP64 sparse direct solution; the solver's
    tolerance of 1e-8 K leaves an error below it, the direct solution's own is
    its backward error times the system's condition (1e-16 x 1e7 of 400 K): bar
    1e-6 K."""
    from hotspot_b200 import STEADY_BICGSTAB
    rng = np.random.default_rng([rows, cols, layers])
    sc = W.scenario_random_chip(workdir, rng, "bc", side=16, chip_layers=layers, steps=1)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    if rows > 8 * cols:
        _narrow(workdir, 4 * cols / rows)
    m, o = hm.from_scenario(sc), OracleModel(sc)
    m.set_solver(FORM_FAST, STEADY_BICGSTAB, steady_tol=1e-8)
    p = m.power_vector(sc.block_power[0] * 0.1)
    s = m.vector()
    for _ in range(2):        # the second from the captured passes
        m.steady(p.copy(), s)
    g, _ = o.steady_direct(p)
    assert np.max(np.abs(m.grid("steady") - g)) <= 1e-6
    m.close()


@pytest.mark.parametrize("rows,cols,layers", [(4, 4, 1), (8, 32, 3), (16, 16, 2), (16, 128, 1), (128, 16, 10), (64, 32, 4),
                                              (128, 128, 1), (256, 128, 1), (32, 256, 2)])
def test_mg_steady_shapes(workdir, rows, cols, layers):
    """The per-layer multigrid at the edges of its parts: one level only, levels
    one CTA of the cluster takes alone, strips of one and of many rows, whole
    passes in the cluster and tiles above it.  Against the FP64 sparse direct
    solution; the solver's tolerance of 1e-8 K leaves an error below it, the
    direct solution's own is its backward error times the system's condition
    (1e-16 x 1e7 of 400 K): bar 1e-6 K."""
    rng = np.random.default_rng([rows, cols, layers])
    sc = W.scenario_random_chip(workdir, rng, "mg", side=16, chip_layers=layers, steps=1)
    sc.config.update(grid_rows=str(rows), grid_cols=str(cols))
    m, o = hm.from_scenario(sc), OracleModel(sc)
    m.set_solver(FORM_FAST, steady_tol=1e-8)
    p = m.power_vector(sc.block_power[0] * 0.1)
    s = m.vector()
    for _ in range(2):        # the second from the captured passes
        m.steady(p.copy(), s)
    g, _ = o.steady_direct(p)
    assert np.max(np.abs(m.grid("steady") - g)) <= 1e-6
    m.close()
