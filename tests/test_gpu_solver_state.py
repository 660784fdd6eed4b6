"""What one solve leaves on a simulation must not reach the next: maps of the water, exchange words, scheduler state."""
import numpy as np
import pytest

from bevy_eulerian_fluid_b200 import _capi as capi
from bevy_eulerian_fluid_b200 import scenes

from .helpers import compare_fields, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,pre", [(768, 80, 2), (768, 80, 3), (520, 120, 2), (2048, 32, 2), (768, 512, 2)])
def test_water_moves_between_solves_of_two_methods(oracle_api, gpu_api, nx, ny, pre):
    """MGPCG, then the water on the other side and iterated V-cycles on the same simulation.  The first three grids are
    at most 256^2 cells and too wide for the V-cycle's cluster, so that their levels run as launches, which skip the
    blocks without water; the V-cycles make a map of level 0 only there."""
    cfg = scenes.base_config(nx, ny)
    sc = scenes.Scene(f"left_{nx}x{ny}", cfg, oneshot=[scenes.aabb_source((-0.4 * nx, -0.2 * ny), (0.1 * nx, 0.3 * ny))])
    P = cfg.projection
    P.method, P.tolerance, P.max_iterations, P.mg_pre = capi.PROJECTION_MGPCG, 1e-5, 12, pre
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(3):
        so, sg = o.step(scenes.DT), g.step(scenes.DT)
    assert not compare_fields(g, o)
    for f in (capi.FIELD_LEVELSET_AIR, capi.FIELD_LEVELSET_AIR1):
        mirrored = np.ascontiguousarray(o.get(f)[:, ::-1])
        for s in (o, g):
            s.set(f, mirrored)
    P.method, P.tolerance = capi.PROJECTION_MULTIGRID, 1e-6
    for s in (o, g):
        s.set_projection(P)
    so, sg = o.step(scenes.DT), g.step(scenes.DT)
    assert (so.pressure_iterations, so.residual_initial) == (sg.pressure_iterations, sg.residual_initial)
    assert not compare_fields(g, o)


def test_every_wait_that_runs_out_is_reported(gpu_api):
    """The tolerance-driven solve with limits of a few polls: whichever CTA's wait runs out, in the first barrier, in an
    exchange or in the last one, when the first CTA may be done already, the solve is an error that names the wait;
    otherwise it is the whole solve.  Aborted solves leave nothing behind: the pressure of before, and exchange words
    that the next solve clears."""
    sc = scenes.coupled(256, tolerance=1e-5, n_per_shape=2)
    sc.cfg.projection.max_iterations, sc.cfg.projection.check_interval = 24, 8
    g = sc.make(gpu_api)
    g.step(sc.dt)
    for stage in range(capi.STAGE_UPDATE_SOLID, capi.STAGE_PROJECTION):
        g.run_stage(stage, sc.dt)
    before = g.get(capi.FIELD_PRESSURE)
    st = g.run_stage(capi.STAGE_PROJECTION, sc.dt)
    want = g.get(capi.FIELD_PRESSURE)
    assert st.pressure_iterations == 24 and not np.array_equal(before, want)
    for limit in [*range(1, 17), 0]:
        for _ in range(6):
            g.set(capi.FIELD_PRESSURE, before)
            g.set_wait_limits(barrier_polls=limit)
            try:
                g.run_stage(capi.STAGE_PROJECTION, sc.dt)
            except capi.EflError as e:
                assert limit and e.status == capi.ERR_CUDA
                assert str(e).endswith(("a grid barrier timed out", "a halo exchange timed out")), str(e)
                assert np.array_equal(g.get(capi.FIELD_PRESSURE), before)
            else:
                assert np.array_equal(g.get(capi.FIELD_PRESSURE), want), limit
    g.close()


def test_batch_waits_as_long_as_a_gang_makes_progress(gpu_api):
    """Two pools of which the device holds one at a time: the CTAs left over wait for the second through the first
    one's whole solve (20000 iterations, 18 ms or more), with a limit of 2000 polls (about 2 ms) that is ample for a
    barrier or an exchange."""
    scs = []
    for i in range(2):
        sc = scenes.batch(1, seed=3 + i, shapes=[(640, 320)]).scenes[0]
        sc.oneshot = [scenes.aabb_source((0.0, 0.0), (320.0, 150.0))]
        sc.cfg.projection.max_iterations, sc.cfg.projection.tolerance = 20000, 1e-14
        scs.append(sc)
    alone = [sc.make(gpu_api) for sc in scs]
    with capi.Batch(gpu_api, [sc.cfg for sc in scs]) as batch:
        scenes.BatchScene("two pools", scs, 0).setup(batch.sims)
        batch.set_wait_limits(2000)
        for _ in range(3):  # the first is the initialisation
            sb = batch.step(scenes.DT)
            sa = [s.step(scenes.DT) for s in alone]
        assert [s.pressure_iterations for s in sb] == [s.pressure_iterations for s in sa] == [20000, 20000]
        for b, a in zip(batch.sims, alone):
            assert not compare_fields(b, a)


def test_batch_reports_the_tiles_of_its_last_solve(gpu_api):
    """A simulation with more water than the device holds streams until the tuner has chosen; without its water the
    solves run by gangs again, and their tiles are reported.  A residual test after every iteration makes the tuner
    choose few iterations per round, other tiles than the gangs'."""
    scs = [scenes.batch(1, seed=100 + i, shapes=[s]).scenes[0] for i, s in enumerate([(1024, 640), (64, 64)])]
    scs[0].oneshot = [scenes.aabb_source((0.0, 0.0), (512.0, 314.0))]
    for sc in scs:
        sc.cfg.projection.max_iterations, sc.cfg.projection.check_interval = 20, 1
    with capi.Batch(gpu_api, [sc.cfg for sc in scs]) as batch:
        scenes.BatchScene("one large", scs, 0).setup(batch.sims)
        for _ in range(8):  # the initialisation, a step that converges at once and four that tune
            batch.step(scenes.DT)
        tuned, cost = batch.tiles()
        assert tuned in [(64, 32, 2), (64, 32, 4), (32, 32, 2), (64, 32, 8)] and all(cost)
        for f in (capi.FIELD_LEVELSET_AIR, capi.FIELD_LEVELSET_AIR1):
            batch.sims[0].set(f, np.full_like(batch.sims[0].get(f), 50.0))
        batch.step(scenes.DT)
        assert batch.tiles()[0] == (64, 32, 4)
        batch.set_tiles(2)
        assert batch.tiles()[0] == (32, 32, 2)
