"""Launches in time slices end like whole runs, whatever is lost on the way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def growing(n, last, rng):
    """Particles whose x grows by px per turn through a 1 m drift, so that the
    10 mm aperture behind it loses them after 0 to ``last`` turns."""
    c = np.zeros((n, 6))
    c[:, 1] = 0.01 / rng.uniform(0.5, last, n) * rng.choice([-1, 1], n)
    return c


@pytest.mark.parametrize('turns', [1000, 2 ** 31 - 1])
@pytest.mark.parametrize('fma', [False, True])
def test_launch_ends_when_every_particle_is_lost(turns, fma):
    """Turns up to INT_MAX stand for "until all are lost"."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    line = u.Line('r', [u.Drift('d', length=1.0),
                        u.Aperture('a', window='x*x + y*y < 1e-4')])
    dp = capi.DeviceProgram(ctx, C.compile_line(line, u.KICK, where=[-1]))
    n = 152 * 12 * 16 + 5
    coords = growing(n, 200, np.random.default_rng(turns % 1000))
    tf = capi.UFO_TRACK_FMA if fma else 0
    got, want = (capi.track(ctx, dp, coords, turns, capi.UFO_MODE_TRACK, tf | f, slots=0)
                 for f in (0, capi.UFO_TRACK_PLAIN))
    assert np.array_equal(got[1], want[1]) and 150 < got[1].max() <= 200
    assert np.array_equal(got[2], want[2], equal_nan=True)


@pytest.mark.parametrize('turns', [2, 37, 4000])
def test_finished_groups_are_passed_over_and_the_others_run_on(turns):
    """A group of 16 whose particles are all lost is handed out no more; groups
    with one survivor, in any of its places, run every turn."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    line = u.Line('r', [u.Quadrupole('q', length=0.2, k1=0.0, slices=4),
                        u.Drift('d', length=0.8), u.Aperture('a', window='x*x + y*y < 1e-4')])
    dp = capi.DeviceProgram(ctx, C.compile_line(line, u.KICK, where=[-1]))
    n = 152 * 16 * 16 + 3
    coords = growing(n, 60, np.random.default_rng(turns))
    alive = np.arange(0, n, 83)  # every fifth group or so, in changing places
    coords[alive, 1] = 0.0
    got, want = (capi.track(ctx, dp, coords, turns, capi.UFO_MODE_TRACK, f, slots=0)
                 for f in (0, capi.UFO_TRACK_PLAIN))
    assert np.array_equal(got[1], want[1]) and np.all(got[1][alive] == turns)
    assert np.array_equal(got[2], want[2], equal_nan=True)


@pytest.mark.parametrize('slices', [4, 7, 8, 13, 15, 29])
def test_constant_divisions_round_subnormal_quotients_correctly(slices):
    """Inner drifts divide by slices - 1; the smallest operands' quotients, ties
    among them, are IEEE division's."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    line = u.Line('r', [u.Sextupole('s', length=4.0, k2=0.0, slices=slices)])
    dp = capi.DeviceProgram(ctx, C.compile_line(line, u.KICK, where=[-1]))
    n = 4000
    rng = np.random.default_rng(slices)
    p = rng.choice([-1.0, 1.0], n) * rng.integers(0, 2000, n) * 2.0 ** -1074
    p[::3] *= 2.0 ** rng.integers(0, 60, len(p[::3]))
    coords = np.zeros((n, 6))
    coords[:, 1], coords[:, 3] = p, p[::-1]
    _, _, got = capi.track(ctx, dp, coords, 1, capi.UFO_MODE_TRACK, 0, slots=0)
    outer = 4.0 / (2 * (1 + slices))
    inner = 4.0 - 2 * outer
    want = p * outer
    for _ in range(slices - 1):
        want = want + (p * inner) / float(slices - 1)
    want = want + p * outer
    assert np.array_equal(got[:, 0], want) and np.array_equal(got[:, 2], want[::-1])


@pytest.mark.parametrize('fma', [False, True])
def test_scans_are_the_same_at_every_tuning(fma):
    """Dynamic-aperture scans with the library's choice of resident warps, and
    tuned, where a full launch of general magnets goes by its size."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C, workloads as W
    ctx = u.context(0)
    prog = C.compile_line(W.c3_ring(u), u.KICK | (u.FMA if fma else 0), where=[-1])
    dp = capi.DeviceProgram(ctx, prog)
    grid = W.c3_grid(128, 128)
    tf = capi.UFO_TRACK_FMA if fma else 0
    want = capi.track(ctx, dp, grid, 12, capi.UFO_MODE_SA, tf | capi.UFO_TRACK_PLAIN, slots=0)
    ctx.reset_tuning()
    try:
        for warps in (None, 1, 7, 16, 32):
            if warps:
                ctx.set_tuning(warps)
            got = capi.track(ctx, dp, grid, 12, capi.UFO_MODE_SA, tf, slots=0)
            assert np.array_equal(got[1], want[1]), warps
            assert np.array_equal(got[2], want[2], equal_nan=True), warps
    finally:
        ctx.reset_tuning()
