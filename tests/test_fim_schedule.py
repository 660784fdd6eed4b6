"""The schedule of k_fim restated on the CPU: 56 x 32 cells per tile with a halo of 20, 10 iterations per launch, the
start state made in the first launch from the advected level set, the active cells as a list, the cells to activate
found beside converged ones, each launch reading the planes of the one before.  After every launch the owned cells equal
the two-phase global iteration's (tests/test_fim_tiling.py states that one), and after the 10 iterations of a step the
oracle's level set.  The kernel itself runs in the GPU tests below and in tests/test_gpu_tiles.py."""
import numpy as np
import pytest

from bevy_eulerian_fluid_b200 import _capi as capi
from bevy_eulerian_fluid_b200 import scenes

from .helpers import compare_fields, make_pair
from .test_fim_tiling import ACTIVE, EPS, LARGE, NONE, SOURCE, F, _init, _iterate, _quad, _sign

TW, TH, HALO = 56, 32, 20


def _tile(S, L, x0, y0, iters):
    """One CTA: the image's cells from the launch's start, large beyond them; its owned cells after `iters`."""
    H, W = S.shape
    xs, ys = range(max(0, x0 - HALO), min(W, x0 + TW + HALO)), range(max(0, y0 - HALO), min(H, y0 + TH + HALO))
    s = {(x, y): S[y, x] for y in ys for x in xs}
    t = dict(s)
    src = {c for c in s if L[c[1], c[0]] == SOURCE}
    act = {c for c in s if L[c[1], c[0]] == ACTIVE}
    work = sorted(act)
    for _ in range(iters):
        if not work:
            break
        conv, nxt = set(), []
        for x, y in work:  # phase A
            p = s[x, y]
            t[x, y] = F(_quad(lambda a, b: F(abs(s.get((a, b), LARGE))), x, y) * _sign(p))
            if abs(F(p - t[x, y])) > EPS:
                nxt.append((x, y))
            else:
                conv.add((x, y))
        beside = {(x + dx, y + dy) for x, y in conv for dx, dy in ((0, 1), (1, 0), (-1, 0), (0, -1))}
        cand = sorted(c for c in beside if c in s and c not in act and c not in src)
        for c in work:
            s[c] = t[c]
        act -= conv
        for x, y in cand:  # phase B
            qn = _quad(lambda a, b: F(abs(t.get((a, b), LARGE))), x, y)
            if F(abs(t[x, y])) > qn:
                frm = next(c for c in ((x, y + 1), (x + 1, y), (x - 1, y), (x, y - 1)) if c in conv)
                s[x, y] = F(qn * _sign(t[frm]))
                act.add((x, y))
                nxt.append((x, y))
        work = nxt
    own = [(x, y) for y in range(y0, min(H, y0 + TH)) for x in range(x0, min(W, x0 + TW))]
    return {c: (s[c], SOURCE if c in src else ACTIVE if c in act else NONE) for c in own}


@pytest.mark.parametrize("nx,ny,iterations", [(96, 64, 10), (120, 72, 25)])
def test_schedule_equals_two_phase_and_oracle(oracle_api, nx, ny, iterations):
    sc = scenes.batch(1, seed=0xC5, shapes=[(nx, ny)]).scenes[0]
    sc.cfg.reinit.fim_iterations = iterations
    sim = sc.make(oracle_api)
    for _ in range(4):
        sim.step(sc.dt)
    S, L = _init(sim.get(capi.FIELD_LEVELSET_AIR1).astype(F))
    Sg, Lg = S.copy(), L.copy()
    for done in range(0, iterations, HALO // 2):
        n = min(HALO // 2, iterations - done)
        _iterate(Sg, Lg, n)
        S2, L2 = S.copy(), L.copy()
        for y0 in range(0, ny, TH):
            for x0 in range(0, nx, TW):
                for (x, y), (v, lab) in _tile(S, L, x0, y0, n).items():
                    S2[y, x], L2[y, x] = v, lab
        S, L = S2, L2
        assert np.array_equal(S, Sg) and np.array_equal(L, Lg), done
    assert np.array_equal(S, sim.get(capi.FIELD_LEVELSET_AIR).astype(F))
    assert np.array_equal(L, sim.get(capi.FIELD_FIM_LABELS))
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("iterations", [10, 35])
def test_late_tiles_read_the_planes_of_the_launch_before(oracle_api, gpu_api, iterations):
    """1280 x 960: 690 tiles, more CTAs than the device holds at once, in one launch and in four, each of which must
    leave the planes that it reads as they are for the CTAs that start late."""
    nx, ny = 1280, 960
    sc = scenes.Scene("dam_break", scenes.base_config(nx, ny),
                      oneshot=[scenes.aabb_source((0.0, -0.2 * ny), (0.5 * nx, 0.3 * ny))])
    sc.cfg.reinit.fim_iterations = iterations
    o, g = make_pair(sc, oracle_api, gpu_api)
    for _ in range(4):
        o.step(scenes.DT)
        g.step(scenes.DT)
    assert not compare_fields(g, o)
