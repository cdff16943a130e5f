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
