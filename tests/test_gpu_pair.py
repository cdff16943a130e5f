"""The two-lane kernel (csrc/pair.cuh) against the one-lane interpreter: the
launches that take it must give the plain kernel's results bit for bit, over
the element models, division forms, special values and table layouts it
accepts."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _beam(n, scale=1.0):
    rng = np.random.default_rng(n)
    c = rng.normal(0, 1, (n, 6)) * np.array([1e-3, 1e-4, 1e-3, 1e-4, 1e-3, 1e-3]) * scale
    c[::5, 2:4] = 0.0  # one plane exactly empty
    return c


def _special(n):
    """Particles with non-finite, huge, tiny and zero coordinates and dp = -1
    beside ordinary ones."""
    c = _beam(n)
    odd = [np.nan, np.inf, -np.inf, 1e300, -1e160, 1e-310, -1e-290, 0.0, -0.0, 0.9]
    k = 0
    for col in (0, 1, 2, 3):
        for v in odd:
            c[k % n, col] = v
            k += 3
    c[1::23, 5] = -1.0
    c[2::29, 5] = -1.0 + 1e-16
    return c


def _rings():
    import ufo_gb300 as u
    from ufo_gb300 import workloads as W
    import os
    alba = u.Lattice(os.path.join(H.HERE, 'golden', 'madx', 'alba.mad')).RING

    def sliced(n):
        """Every teapot element type with n slices (inner drifts divide by n - 1)."""
        q = u.Quadrupole('q', length=0.3, k1=1.1, slices=n, dx=1e-4)
        s = u.Sextupole('s', length=0.2, k2=30.0, slices=n, dy=-2e-4)
        b = u.Sbend('b', length=1.1, angle=0.1, k1=-0.3, e1=0.02, slices=n)
        g = u.Quadrupole('g', length=0.25, k1=-1.1, slices=n, dkn=[0, 0, 3.0, 0, 2e4, 1e6, 1e8],
                         dks=[1e-5, 0.01, 0, 50.0])
        o = u.Octupole('o', length=0.1, k3=500.0, slices=n)
        return u.Line('r', [q, u.Drift('d', length=0.7), s, b, u.Drift('e', length=0.4), g, o])

    mixed = u.Line('m', [u.Drift('d', length=0.3), u.Wire('w', x=0.01, y=0.002, k=1e-6),
                         u.Quadrupole('q', length=0.2, k1=1.0, slices=4),
                         u.Aperture('a', window='fabs(x) < 0.02 && fabs(y) < 0.01'),
                         u.Multipole('m', knl=[0, 0.1, 2.0], ksl=[1e-4]),
                         u.Multipole('n', knl=[0, 0.1]), u.Multipole('t', knl=[0, 0, 4.0]),
                         u.Marker('z'), u.Sbend('b', length=0.5, angle=0.05, slices=4),
                         u.Aperture('c', window='x*x + y*y < 1e-3')])
    out = {'c1': (W.c1_ring(u), u.KICK), 'c3': (W.c3_ring(u), u.KICK),
           'c5': (W.c5_ring(u), u.KICK), 'alba_kick': (alba, u.KICK),
           'alba_thick': (alba, 0), 'alba_achromatic': (alba, u.ACHROMATIC),
           'alba_linear': (alba, u.LINEAR | u.ACHROMATIC), 'c1_thick': (W.c1_ring(u), 0),
           'alba_fived': (alba, u.FIVED), 'mixed': (mixed, u.KICK), 'mixed_thick': (mixed, 0)}
    for n in (1, 2, 3, 4, 5, 6, 7, 8, 13, 16, 29):
        out[f'slices{n}'] = (sliced(n), u.KICK)
    return out


NAMES = ['c1', 'c3', 'c5', 'alba_kick', 'alba_thick', 'alba_achromatic', 'alba_linear', 'c1_thick',
         'alba_fived', 'mixed', 'mixed_thick'] + [f'slices{n}' for n in
                                                   (1, 2, 3, 4, 5, 6, 7, 8, 13, 16, 29)]


def _same(a, b):
    return all(np.array_equal(x, y, equal_nan=x.dtype.kind == 'f') for x, y in zip(a, b))


@pytest.mark.parametrize('name', NAMES)
def test_two_lane_kernel_is_the_one_lane_interpreter(name):
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    line, flags = _rings()[name]
    ctx = u.context(0)
    where = [1.5, 2, -1]
    turns = 2 if name == 'c5' else 5
    for fma in (0, u.FMA):
        prog = C.compile_line(line, flags | fma, where=where)
        dp = capi.DeviceProgram(ctx, prog)
        tf = capi.UFO_TRACK_FMA if fma else 0
        for coords in (_beam(1), _beam(17), _special(333), _beam(1000, 10.0)):
            for mode in (capi.UFO_MODE_TRACK, capi.UFO_MODE_SA):
                slots = 3 * turns
                one = capi.track(ctx, dp, coords, turns, mode, tf | capi.UFO_TRACK_PLAIN,
                                 slots=slots)
                two = capi.track(ctx, dp, coords, turns, mode, tf, slots=slots)
                assert _same(one, two), (fma, len(coords), mode)


@pytest.mark.parametrize('slices', [4, 7, 8, 13, 15])
def test_constant_divisions_are_correctly_rounded(slices):
    """Inner drifts divide by slices - 1 (3, 6, 7, 12, 14): many random
    operands against the one-lane code's division, and the first slice's
    quotient against IEEE division on the host through one drift-only element."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    line = u.Line('r', [u.Sextupole('s', length=0.2, k2=0.0, slices=slices)])
    dp = capi.DeviceProgram(ctx, C.compile_line(line, u.KICK, where=[-1]))
    rng = np.random.default_rng(slices)
    n = 200_000
    coords = np.zeros((n, 6))
    for j in range(4):
        coords[:, j] = rng.choice([-1, 1], n) * np.exp2(rng.uniform(-900, 300, n)) \
            * rng.uniform(1, 2, n)
    _, _, got = capi.track(ctx, dp, coords, 1, capi.UFO_MODE_TRACK, 0, slots=0)
    L = 0.2
    outer = L / (2 * (1 + slices))
    inner = L - 2 * outer
    ref = coords.copy()
    with np.errstate(all='ignore'):
        for q in (0, 2):
            x, p = coords[:, q], coords[:, q + 1]
            x = x + p * outer
            for _ in range(slices - 1):
                x = x + (p * inner) / float(slices - 1)
            ref[:, q] = x + p * outer
    assert np.array_equal(got[:, :4], ref[:, :4])


def test_seeds_turn_counts_and_new_tables():
    """Per-particle rows and turn counts, and a replaced table whose constants
    share other cache fields, against the one-lane code."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    line, _ = _rings()['alba_thick']
    flat = line.flatten()
    at = [i for i, e in enumerate(flat) if type(e).__name__ in ('Quadrupole', 'Sbend')][:40]
    params = [(i, 'k1') for i in at]
    base = np.array([flat[i].k1 for i in at])
    rng = np.random.default_rng(0)
    same = np.repeat(base[None], 5, axis=0)
    varied = same * (1 + 1e-3 * rng.standard_normal(same.shape))
    coords = _beam(251)
    seed = rng.integers(0, 5, 251).astype(np.int32)
    pturns = rng.integers(0, 9, 251).astype(np.int32)
    dp = capi.DeviceProgram(ctx, C.compile_line(line, 0, params, [-1], seed_values=same))
    for rows in (same, varied, same):
        dp.set_table(C.compile_line(line, 0, params, [-1], seed_values=rows).table)
        out = [capi.track(ctx, dp, coords, 9, capi.UFO_MODE_TRACK, f, seed=seed, pturns=pturns,
                          slots=0)[1:] for f in (capi.UFO_TRACK_PLAIN, 0)]
        assert _same(*out)


def test_tables_that_change_the_two_lane_form():
    """Strengths too small for the two-lane form send their elements through the
    one-lane code; tables may switch between the two."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    line, flags = _rings()['c1']
    at = [i for i, e in enumerate(line.flatten()) if type(e).__name__ == 'Quadrupole']
    params = [(i, 'k1') for i in at]
    coords = _beam(100)
    plain = np.full((1, len(at)), 1.1)
    tiny = plain.copy()
    tiny[0, ::2] = 1e-300
    tiny[0, 1::4] = 1e300
    for fma in (0, u.FMA):
        tf = capi.UFO_TRACK_FMA if fma else 0
        dp = capi.DeviceProgram(ctx, C.compile_line(line, flags | fma, params, [-1],
                                                    seed_values=plain))
        for rows in (plain, tiny, plain):
            dp.set_table(C.compile_line(line, flags | fma, params, [-1], seed_values=rows).table)
            out = [capi.track(ctx, dp, coords, 3, capi.UFO_MODE_TRACK, tf | f, slots=0)[1:]
                   for f in (capi.UFO_TRACK_PLAIN, 0)]
            assert _same(*out)


def test_graph_of_a_thick_batch_keeps_its_cache():
    """A captured graph goes on using the coefficient cache while larger
    launches and new tables of the same program come and go."""
    import ufo_gb300 as u
    from ufo_gb300 import capi
    ctx = u.context(0)
    line, _ = _rings()['alba_thick']
    at = [i for i, e in enumerate(line.flatten()) if type(e).__name__ == 'Quadrupole'][:6]
    k1 = np.array([line.flatten()[i].k1 for i in at])
    rng = np.random.default_rng(1)
    rows = k1 * (1 + 1e-3 * rng.standard_normal((3, len(at))))
    b = u.TrackBatch(line, [(i, 'k1') for i in at], rows, [20, 7, 33], [4, 6, 5], flags=0)
    b.coords[:] = _beam(60)
    first = [v.copy() for v in b.run()]
    plain = [v.copy() for v in b.run_plain()]
    assert _same(first, plain)
    b.upload()
    b.capture()
    big = np.repeat(_beam(60), 700, axis=0)
    capi.track(ctx, b.dprog, big, 1, capi.UFO_MODE_TRACK, 0, slots=0)
    b.dprog.set_table(b.prog.table * 1.0)
    b.launch()
    assert _same(first, b.download())


@pytest.mark.parametrize('name', ['c1', 'alba_kick', 'mixed'])
@pytest.mark.parametrize('n', [1, 3, 700])
def test_closed_orbits_of_lane_pairs_are_the_one_thread_searchs(name, n):
    """The four-trial search (one and four orbits per warp) against the
    one-thread search, which batches beyond 64 orbits per SM take: regular
    starts, a start on the orbit (equal residuals), far and non-finite ones."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    line, flags = _rings()[name]
    ctx = u.context(0)
    at = [i for i, e in enumerate(line.flatten()) if type(e).__name__ == 'Quadrupole'][:3]
    params = [(i, 'dx') for i in at]
    rows = np.random.default_rng(5).normal(0, 1e-4, (7, len(at)))
    rows[0] = 0.0  # the orbit is exactly zero
    dp = capi.DeviceProgram(ctx, C.compile_line(line, flags, params, [], seed_values=rows))
    start = _beam(n)[:, :4] * 0.1
    start[0] = 0.0
    if n > 3:
        start[5] = 0.5
        start[6, 1] = np.nan
        start[7, 2] = np.inf
    seed = (np.arange(n) % 7).astype(np.int32)

    def orbits(st, sd, steps):
        out = np.empty_like(st)
        capi.check(capi.load().ufo_closed_orbit(ctx.handle, dp.handle, capi.ptr(st),
                                                capi.ptr(sd), len(st), steps, capi.ptr(out)))
        return out
    import torch
    many = 64 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    reps = -(-many // n)
    for steps in (0, 1, 37):
        got = orbits(start, seed, steps)
        ref = orbits(np.tile(start, (reps, 1)), np.tile(seed, reps), steps)[:n]
        assert np.array_equal(got, ref, equal_nan=True)


@pytest.mark.parametrize('name', ['c1', 'alba_thick', 'mixed'])
@pytest.mark.parametrize('n,turns', [(152 * 8 * 16 + 1, 2), (40_000, 5), (50_001, 37)])
def test_time_slices_give_whole_runs(name, n, turns):
    """Launches of more particles than stay resident are cut into slices of
    turns; every particle, special values and observations included, ends as in
    the plain kernel."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    line, flags = _rings()[name]
    if name == 'alba_thick' and turns > 5:
        turns = 3
    ctx = u.context(0)
    coords = np.concatenate([_special(333), _beam(n - 333, 3.0)])
    seed = np.zeros(n, np.int32)
    for fma in (0, u.FMA):
        dp = capi.DeviceProgram(ctx, C.compile_line(line, flags | fma, where=[2, -1]))
        tf = capi.UFO_TRACK_FMA if fma else 0
        out = [capi.track(ctx, dp, coords, turns, capi.UFO_MODE_TRACK, tf | f, seed=seed,
                          slots=2 * (turns // 2), every=2)
               for f in (capi.UFO_TRACK_PLAIN, 0)]
        assert _same(*out), fma
