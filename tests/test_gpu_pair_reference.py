"""The two-lane kernels against references that never take them: closed orbits
against the search on the host over one-turn plain launches, misaligned general
magnets and launches in place against the plain kernel."""
import numpy as np
import pytest

from test_gpu_pair import _beam, _rings, _same, _special

pytestmark = pytest.mark.gpu


def search(v, steps):
    """The Nelder-Mead search of one orbit (ufo/co.py:18-124): yields a vertex, is
    sent its residual, returns the best vertex after ``steps`` steps."""
    sx = [list(v) for _ in range(5)]
    for j in range(4):
        sx[j + 1][j] += 1e-4
    y = []
    for i in range(5):
        y.append((yield sx[i]))
    psum = [sum_of(sx, j) for j in range(4)]

    def trial(fac):
        f1 = (1.0 - fac) / 4.0
        f2 = f1 - fac
        t = [psum[j] * f1 - sx[ihi][j] * f2 for j in range(4)]
        yt = yield t
        if yt < y[ihi]:
            y[ihi] = yt
            for j in range(4):
                psum[j] = psum[j] + (t[j] - sx[ihi][j])
                sx[ihi][j] = t[j]
        return yt
    it = 0
    while True:
        ilo = 1
        ihi, inhi = (1, 2) if y[1] > y[2] else (2, 1)
        for i in range(5):
            if y[i] < y[ilo]:
                ilo = i
            if y[i] > y[ihi]:
                inhi, ihi = ihi, i
            elif y[i] > y[inhi] and i != ihi:
                inhi = i
        if it >= steps:
            return sx[ilo]
        yt = yield from trial(-1.0)
        it += 1
        if yt <= y[ilo]:
            yield from trial(2.0)
        elif yt >= y[inhi]:
            save = y[ihi]
            yt = yield from trial(0.5)
            if yt >= save:
                for i in range(5):
                    if i != ilo:
                        sx[i] = [(sx[i][j] + sx[ilo][j]) * 0.5 for j in range(4)]
                        y[i] = yield sx[i]
                it += 4
                psum[:] = [sum_of(sx, j) for j in range(4)]


def sum_of(sx, j):
    s = 0.0
    for i in range(5):
        s = s + sx[i][j]
    return s


def host_orbits(one_turn, start, steps):
    """All orbits' searches side by side: one launch per round of vertices."""
    runs = [search([float(x) for x in v], steps) for v in start]
    out = np.empty_like(start)
    ask = {k: next(g) for k, g in enumerate(runs)}
    while ask:
        at = np.array(list(ask.values()))
        with np.errstate(all='ignore'):
            d = at - one_turn(at, np.array(list(ask)))
            d = d * d
            res = ((d[:, 0] + d[:, 1]) + d[:, 2]) + d[:, 3]
        new = {}
        for k, r in zip(ask, res.tolist()):
            try:
                new[k] = runs[k].send(r)
            except StopIteration as end:
                out[k] = end.value
        ask = new
    return out


@pytest.mark.parametrize('name', ['c1', 'c1_thick', 'alba_kick', 'alba_thick', 'mixed',
                                  'mixed_thick'])
@pytest.mark.parametrize('n', [3, 700])
def test_closed_orbits_are_the_host_searchs(name, n):
    """One orbit per warp (n up to 4 per SM) and four, on cached thick and fringe
    coefficients as on kicks: misaligned rows, a start on the orbit, far and
    non-finite starts."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    line, flags = _rings()[name]
    ctx = u.context(0)
    at = [i for i, e in enumerate(line.flatten()) if type(e).__name__ == 'Quadrupole'][:3]
    rows = np.random.default_rng(5).normal(0, 1e-4, (7, len(at)))
    rows[0] = 0.0
    dp = capi.DeviceProgram(ctx, C.compile_line(line, flags, [(i, 'dx') for i in at], [],
                                                seed_values=rows))
    start = _beam(n)[:, :4] * 0.1
    start[0] = 0.0
    if n > 3:
        start[5] = 0.5
        start[6, 1] = np.nan
        start[7, 2] = np.inf
    seed = (np.arange(n) % 7).astype(np.int32)

    def one_turn(v, which):
        c = np.zeros((len(v), 6))
        c[:, :4] = v
        return capi.track(ctx, dp, c, 1, capi.UFO_MODE_TRACK, capi.UFO_TRACK_PLAIN,
                          seed=seed[which], slots=0)[2][:, :4]
    for steps in (0, 1, 23):
        got = np.empty_like(start)
        capi.check(capi.load().ufo_closed_orbit(ctx.handle, dp.handle, capi.ptr(start),
                                                capi.ptr(seed), n, steps, capi.ptr(got)))
        assert np.array_equal(got, host_orbits(one_turn, start, steps), equal_nan=True), steps


@pytest.mark.parametrize('dx,dy', [(1e-4, 0.0), (0.0, -2e-4), (1e-4, -2e-4)])
@pytest.mark.parametrize('edge', [0.0, 0.03])
def test_general_magnets_misaligned_in_one_plane(dx, dy, edge):
    """The shifts around a general magnet run with it, with and without an edge in
    between, in either plane alone and in both; neighbours shifted differently."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    err = dict(dkn=[0, 0, 3.0, 0, 2e4], dks=[1e-5, 0.01])
    g = u.Quadrupole('g', length=0.25, k1=-1.1, slices=4, dx=dx, dy=dy, **err)
    b = u.Sbend('b', length=1.1, angle=0.1, k1=0.3, e1=edge, e2=-edge, slices=4, dx=dx, dy=dy,
                **err)
    h = u.Quadrupole('h', length=0.25, k1=1.1, slices=3, dx=-dy, dy=dx, **err)
    z = u.Quadrupole('z', length=0.25, k1=1.1, slices=1, dx=dx, **err)
    line = u.Line('r', [g, b, h, u.Drift('d', length=0.3), h, g, z, z, b, u.Drift('e', length=0.2)])
    for flags, tf in ((u.KICK, 0), (u.KICK | u.FMA, capi.UFO_TRACK_FMA)):
        dp = capi.DeviceProgram(ctx, C.compile_line(line, flags, where=[3, -1]))
        for coords in (_beam(17), _special(333)):
            out = [capi.track(ctx, dp, coords, 4, capi.UFO_MODE_TRACK, tf | f, slots=8)
                   for f in (0, capi.UFO_TRACK_PLAIN)]
            assert _same(*out)


@pytest.mark.parametrize('name', ['c1', 'alba_thick', 'c3'])
@pytest.mark.parametrize('n', [300, 40_000])
def test_final_coordinates_may_replace_the_initial_ones(name, n):
    """d_final = d_coords, whole runs and slices."""
    import torch
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    line, flags = _rings()[name]
    ctx = u.context(0)
    coords = np.concatenate([_special(min(n, 333)), _beam(max(1, n - 333), 3.0)])[:n]
    dp = capi.DeviceProgram(ctx, C.compile_line(line, flags, where=[-1]))
    turns = 3 if name != 'c1' else 40
    want = capi.track(ctx, dp, coords, turns, capi.UFO_MODE_TRACK, capi.UFO_TRACK_PLAIN, slots=0)
    c = torch.from_numpy(coords).to('cuda:0')
    lost = torch.empty(n, dtype=torch.int32, device='cuda:0')
    torch.cuda.synchronize()
    capi.check(capi.load().ufo_track_device(
        ctx.handle, dp.handle, capi.ptr(c.data_ptr()), None, None, n, turns, capi.UFO_MODE_TRACK,
        0, 0, 1, None, capi.ptr(lost.data_ptr()), capi.ptr(c.data_ptr()), None))
    torch.cuda.synchronize()
    assert np.array_equal(lost.cpu().numpy().view(np.uint32), want[1])
    assert np.array_equal(c.cpu().numpy(), want[2], equal_nan=True)
