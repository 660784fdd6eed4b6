"""The tiled stage kernels at the sizes where a tile, its halo or its masks end, against the CPU oracle, bit for bit:
the fast iterative method (56 x 32 cells with a 20-cell halo, 10 iterations per launch) and the velocity
extrapolation (32 x 32 faces with a 10-face halo)."""
import numpy as np
import pytest

from bevy_eulerian_fluid_b200 import _capi as capi
from bevy_eulerian_fluid_b200 import scenes

from .helpers import compare_fields, make_pair

pytestmark = pytest.mark.gpu


def _splash(nx, ny, iterations=10):
    """Water on the left, two droplets (one across a tile corner) and a jet: interfaces in every part of the grid."""
    cfg = scenes.base_config(nx, ny)
    cfg.reinit.fim_iterations = iterations
    r = 0.11 * min(nx, ny)
    once = [scenes.aabb_source((-0.25 * nx, -0.2 * ny), (0.25 * nx, 0.3 * ny)),
            scenes.circle_source((56 - 0.5 * nx, 0.5 * ny - 32), r), scenes.circle_source((0.3 * nx, 0.2 * ny), r)]
    jet = [scenes.circle_source((0.1 * nx, 0.3 * ny), 0.06 * min(nx, ny), velocity=(25.0, -40.0))]
    return scenes.Scene(f"splash_{nx}x{ny}", cfg, oneshot=once, continuous=jet)


@pytest.mark.parametrize("nx,ny,iterations", [(64, 64, 10), (56, 32, 10), (112, 64, 1), (120, 72, 9), (168, 40, 11),
                                              (64, 200, 20), (200, 136, 25), (128, 96, 0), (16, 16, 10), (24, 440, 10),
                                              (704, 448, 10)])
def test_tiled_stages_bit_exact(oracle_api, gpu_api, nx, ny, iterations):
    o, g = make_pair(_splash(nx, ny, iterations), oracle_api, gpu_api)
    for _ in range(7):
        o.step(scenes.DT)
        g.step(scenes.DT)
    assert not compare_fields(g, o)


@pytest.mark.parametrize("nx,ny", [(200, 136), (128, 64)])
def test_extrapolation_reads_flags_outside_the_dispatch(oracle_api, gpu_api, nx, ny):
    """Faces beyond floor(n / 64) * 64 keep whatever flags they hold, and the sweeps read them."""
    o, g = make_pair(_splash(nx, ny), oracle_api, gpu_api)
    rng = np.random.default_rng(5)
    for s in (o, g):
        s.step(scenes.DT)
        s.step(scenes.DT)
    for f in (capi.FIELD_U_VALID, capi.FIELD_V_VALID):
        flags = (rng.random(o.get(f).shape) < 0.3).astype(np.int32)
        o.set(f, flags)
        g.set(f, flags)
    for _ in range(3):
        for s in (o, g):
            s.step(scenes.DT)
    assert not compare_fields(g, o)


@pytest.mark.parametrize("method,tolerance", [(capi.PROJECTION_MULTIGRID, 0.0), (capi.PROJECTION_MULTIGRID, 1e-3),
                                              (capi.PROJECTION_MGPCG, 1e-5)])
@pytest.mark.parametrize("nx,ny", [(64, 64), (16, 16), (136, 88), (24, 200), (256, 256), (1024, 32), (328, 264),
                                   (512, 640)])
def test_v_cycle_levels_bit_exact(oracle_api, gpu_api, nx, ny, method, tolerance):
    """The lower levels of a V-cycle in one cluster: slabs of every height, odd coarse sizes, levels gathered in one
    CTA, f32 (one cycle, the preconditioner) and f64 (iterated cycles)."""
    sc = _splash(nx, ny)
    sc.cfg.projection.method = method
    sc.cfg.projection.tolerance = tolerance
    sc.cfg.projection.max_iterations = 12
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(4):
        so, sg = o.step(scenes.DT), g.step(scenes.DT)
        assert so.pressure_iterations == sg.pressure_iterations
    assert not compare_fields(g, o)


@pytest.mark.parametrize("nx,ny", [(16, 16), (32, 64), (40, 24), (200, 136), (96, 320)])
def test_jacobi_tiles_bit_exact(oracle_api, gpu_api, nx, ny):
    """Ten Jacobi iterations per launch on 32 x 32 tiles with a 10-cell halo."""
    sc = _splash(nx, ny)
    sc.cfg.projection.method = capi.PROJECTION_JACOBI
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(5):
        o.step(scenes.DT)
        g.step(scenes.DT)
    assert not compare_fields(g, o)


def test_batch_gangs_of_every_kind(gpu_api):
    """A batch with a simulation without water, one with more tiles of water than the device holds (streamed), ragged
    ones, ones of a single tile, and more simulations than fit at once: each as its own solve, bit for bit."""
    shapes = [(128, 128), (1024, 640), (64, 64), (200, 72), (16, 16), (256, 256), (520, 96)] + [(96, 64)] * 30
    scs = []
    for i, (nx, ny) in enumerate(shapes):
        sc = scenes.batch(1, seed=100 + i, shapes=[(nx, ny)]).scenes[0]
        if i == 0:
            sc.oneshot = []
        if i == 1:  # full of water
            sc.oneshot = [scenes.aabb_source((0.0, 0.0), (0.5 * nx, 0.49 * ny))]
        sc.cfg.projection.max_iterations = 400
        scs.append(sc)
    alone = [sc.make(gpu_api) for sc in scs]
    with capi.Batch(gpu_api, [sc.cfg for sc in scs]) as batch:
        scenes.BatchScene("kinds", scs, 0).setup(batch.sims)
        for _ in range(4):
            sb = batch.step(scenes.DT)
            sa = [s.step(scenes.DT) for s in alone]
            assert [(x.pressure_iterations, x.converged) for x in sb] == [(x.pressure_iterations, x.converged) for x in sa]
        for i, (g, a) in enumerate(zip(batch.sims, alone)):
            assert not compare_fields(g, a), shapes[i]


@pytest.mark.parametrize("nx,ny", [(64, 64), (16, 200), (200, 136), (352, 320), (1024, 256)])
def test_solve_on_tiles_with_water(oracle_api, gpu_api, nx, ny):
    """The tolerance-driven solve on the tiles with water only (32 x 32; 64 x 32 where those are too many)."""
    sc = _splash(nx, ny)
    sc.cfg.projection.tolerance = 1e-4
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(4):
        so, sg = o.step(scenes.DT), g.step(scenes.DT)
        assert so.pressure_iterations == sg.pressure_iterations
    assert not compare_fields(g, o)


@pytest.mark.parametrize("nx,ny", [(16, 16), (104, 72), (48, 200), (264, 64)])
def test_weight_gradients_of_ragged_images(gpu_api, nx, ny):
    """The weight- and bias-gradient GEMMs where the last block of 64 pixels, the last chunk and the last tile of 128
    rows are partial; bounds as for the network's other gradients (ReLU and bf16 flips reach a few percent)."""
    from oracle import unet_ref

    from .test_unet import _random_case, _rel
    params, feats, target, mask = _random_case(21, n=ny, nx=nx)
    net = capi.UNet(gpu_api, nx, ny)
    net.set_params(params)
    loss, g = net.gradients(feats, target, mask)
    ref = unet_ref.Net(params)
    ref.forward(feats)
    rloss, rg = ref.backward(target, mask)
    cos = float(g.astype(np.float64) @ rg / (np.linalg.norm(g) * np.linalg.norm(rg)))
    assert loss == pytest.approx(rloss, rel=2e-3) and cos > 0.998 and _rel(g, rg) < 0.06
    off = 0
    for ci, co, _ in unet_ref.SPEC:  # each layer's bias gradient: a row of its own in the GEMM
        off += 9 * ci * co
        assert _rel(g[off:off + co], rg[off:off + co]) < 0.08
        off += co


@pytest.mark.parametrize("nx,ny,iterations", [(16, 16, 1), (32, 16, 5), (64, 64, 6), (72, 40, 10), (200, 136, 11),
                                              (256, 256, 20), (384, 192, 4), (392, 200, 20), (512, 512, 9)])
def test_fixed_count_sweeps_on_both_tiles(oracle_api, gpu_api, nx, ny, iterations):
    """Fixed-count red-black sweeps in one launch: 32 x 16 tiles, exchanged every 5 iterations, where one per SM holds
    the grid, else 64 x 32 every 4."""
    sc = _splash(nx, ny)
    sc.cfg.projection.gs_iterations = iterations
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(5):
        o.step(scenes.DT)
        g.step(scenes.DT)
    assert not compare_fields(g, o)


@pytest.mark.parametrize("nx,ny,interval,limit", [(64, 32, 1, 7), (72, 40, 4, 40), (96, 96, 8, 37), (200, 136, 9, 100),
                                                  (136, 264, 16, 64), (264, 72, 33, 200), (640, 512, 20, 45)])
def test_exchanges_of_every_check_interval(oracle_api, gpu_api, nx, ny, interval, limit):
    """The persistent solve's exchanges by tagged words: checks more often than exchanges, on them and between them, a
    limit that cuts an interval short, one tile and many, and a second solve over the words of the first."""
    sc = _splash(nx, ny)
    sc.cfg.projection.tolerance = 1e-6
    sc.cfg.projection.check_interval = interval
    sc.cfg.projection.max_iterations = limit
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(4):
        so, sg = o.step(scenes.DT), g.step(scenes.DT)
        assert (so.pressure_iterations, so.converged) == (sg.pressure_iterations, sg.converged)
    assert not compare_fields(g, o)


def test_exchanges_of_the_larger_tiles(oracle_api, gpu_api):
    """More 32 x 32 tiles with water than the device holds: 64 x 32 tiles of 4 x 2 blocks, an exchange every 4."""
    nx, ny = 704, 360
    sc = _splash(nx, ny)
    sc.oneshot = [scenes.aabb_source((0.0, 0.0), (0.5 * nx, 0.45 * ny))]
    sc.cfg.projection.tolerance = 1e-6
    sc.cfg.projection.max_iterations = 50
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(3):
        so, sg = o.step(scenes.DT), g.step(scenes.DT)
        assert (so.pressure_iterations, so.converged) == (sg.pressure_iterations, sg.converged)
    assert not compare_fields(g, o)


@pytest.mark.parametrize("nx,ny,pre,post", [(328, 264, 2, 2), (264, 328, 1, 2), (1024, 72, 2, 1), (520, 136, 1, 1),
                                            (328, 264, 3, 2), (328, 264, 2, 0), (768, 512, 2, 2)])
@pytest.mark.parametrize("method,tolerance", [(capi.PROJECTION_MULTIGRID, 0.0), (capi.PROJECTION_MULTIGRID, 1e-3)])
def test_smoothing_passes_bit_exact(oracle_api, gpu_api, nx, ny, pre, post, method, tolerance):
    """A level's one or two smoothing iterations in one pass over 32 x 32 tiles with a halo of 4, in f32 and f64, and
    the launches per half-sweep for other counts."""
    sc = _splash(nx, ny)
    sc.cfg.projection.method = method
    sc.cfg.projection.tolerance = tolerance
    sc.cfg.projection.mg_pre, sc.cfg.projection.mg_post = pre, post
    sc.cfg.projection.max_iterations = 5
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(3):
        so, sg = o.step(scenes.DT), g.step(scenes.DT)
        assert so.pressure_iterations == sg.pressure_iterations
    assert not compare_fields(g, o)
