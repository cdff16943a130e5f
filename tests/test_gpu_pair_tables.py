"""The two-lane kernel's coefficient cache over captures and new tables: every
launch gives the plain kernel's results, whatever entries the constants share."""
import os

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def alba():
    import ufo_gb300 as u
    return u.Lattice(os.path.join(H.HERE, 'golden', 'madx', 'alba.mad')).RING


def beam(n, seed=0):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (n, 6)) * np.array([1e-3, 1e-4, 1e-3, 1e-4, 1e-3, 1e-3])


def same(a, b):
    return all(np.array_equal(x, y, equal_nan=x.dtype.kind == 'f') for x, y in zip(a, b))


def thick_batch(rows, line=None):
    """A thick batch whose magnets' strengths are the columns of ``rows``, and a
    function giving the table of other strengths."""
    import ufo_gb300 as u
    from ufo_gb300 import compiler as C
    line = line or alba()
    at = [i for i, e in enumerate(line.flatten())
          if type(e).__name__ in ('Quadrupole', 'Sbend')][:rows.shape[1]]
    params = [(i, 'k1') for i in at]
    b = u.TrackBatch(line, params, rows, [20, 7, 33], [4, 6, 5], flags=0)
    b.coords[:] = beam(60)
    return b, lambda k1: C.compile_line(line, 0, params, [], seed_values=k1).table


def plain(b):
    from ufo_gb300 import capi
    return capi.track(b.ctx, b.dprog, b.coords, int(b.turns.max()), b.mode,
                      capi.UFO_TRACK_PLAIN, seed=b.seed, pturns=b.pturns, slots=0)[:0:-1]


@pytest.mark.parametrize('captured', ['equal', 'individual'])
def test_captured_thick_batch_takes_tables_that_share_other_entries(captured):
    """A launch captured with equal strengths, then individual ones (more entries
    than the cache has), and the reverse: replay and direct launch both track the
    table that stands."""
    rng = np.random.default_rng(3)
    magnets = [e for e in alba().flatten() if type(e).__name__ in ('Quadrupole', 'Sbend')][:40]
    equal = np.array([[e.k1 for e in magnets]] * 3)  # families of equal magnets
    individual = equal * (1 + 1e-3 * rng.standard_normal(equal.shape))
    tables = {'equal': equal, 'individual': individual}
    b, table = thick_batch(tables[captured])
    b.upload()
    b.capture()
    other = 'individual' if captured == 'equal' else 'equal'
    seen = []
    for name in (captured, other, captured):
        b.dprog.set_table(table(tables[name]))
        want = plain(b)
        for graph in (True, False):
            b.launch(graph=graph)
            assert same(b.download(), want), (name, graph)
        seen.append(want[0])
    assert np.isfinite(seen[0]).all() and not np.array_equal(seen[0], seen[1])
    assert np.array_equal(seen[0], seen[2])


def test_a_callers_own_capture_may_come_first():
    """The first launch of a thick program in the caller's capture, where nothing
    can be allocated, then larger launches, a second capture that holds the cache
    they left, and new tables."""
    import torch
    rng = np.random.default_rng(4)
    magnets = [e for e in alba().flatten() if type(e).__name__ in ('Quadrupole', 'Sbend')][:12]
    rows = np.array([[e.k1 for e in magnets]] * 3)
    b, table = thick_batch(rows)
    b.upload()
    want = plain(b)
    stream = torch.cuda.Stream()
    graphs = []
    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            b.launch(stream=stream.cuda_stream, graph=False)
        graphs.append(g)
        b._dev['final'].zero_()
        g.replay()
        assert same(b.download(), want)
        b._dev['final'].zero_()
        b.launch(graph=False)
        assert same(b.download(), want)
    other = rows * (1 + 1e-3 * rng.standard_normal(rows.shape))
    b.dprog.set_table(table(other))
    want = plain(b)
    for g in graphs:
        b._dev['final'].zero_()
        g.replay()
        assert same(b.download(), want)


def test_a_first_launch_beside_a_capture_leaves_it_alone():
    """A thick program's first launch allocates; a capture of the same thread on
    another stream, in the mode that forbids that, goes on."""
    import torch
    b, _ = thick_batch(np.full((3, 1), 1.4))
    b.upload()
    x = torch.zeros(8, device='cuda:0')
    torch.cuda.synchronize()
    side, work = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side, capture_error_mode='global'):
        x += 1
        b.launch(stream=work.cuda_stream, graph=False)
        x += 1
    work.synchronize()
    g.replay()
    got = b.download()
    assert float(x.sum()) == 16.0
    assert same(got, plain(b))


def test_graphs_outlive_larger_launches_and_one_another():
    """Caches grow past a live graph, and when the last graph is gone a table may
    need more entries again."""
    from ufo_gb300 import capi
    rng = np.random.default_rng(5)
    magnets = [e for e in alba().flatten() if type(e).__name__ in ('Quadrupole', 'Sbend')]
    equal = np.array([[e.k1 for e in magnets]] * 3)
    individual = equal * (1 + 1e-3 * rng.standard_normal(equal.shape))
    b, table = thick_batch(equal)
    b.upload()
    b.capture()
    for rows in (equal, individual, equal):
        b.dprog.set_table(table(rows))
        want = plain(b)
        b.launch()
        assert same(b.download(), want)
        for n in (3000, 40_000, 80_000):  # whole runs, slices, whole runs again
            c = np.tile(b.coords, (-(-n // 60), 1))[:n]
            out = [capi.track(b.ctx, b.dprog, c, 2, capi.UFO_MODE_TRACK, f, slots=0)[1:]
                   for f in (0, capi.UFO_TRACK_PLAIN)]
            assert same(*out), n
        b.launch()
        assert same(b.download(), want)
    b.destroy_graph()
    b.dprog.set_table(table(individual))
    want = plain(b)
    b.capture()
    for graph in (True, False):
        b.launch(graph=graph)
        assert same(b.download(), want)


@pytest.mark.parametrize('rows', [2, 3000])
@pytest.mark.parametrize('what', ['strength', 'division', 'entry'])
def test_one_row_apart_is_seen_in_small_and_large_tables(rows, what):
    """Tables are looked through on the host or, when large, on the GPU: a last
    row whose strengths, inner-drift divisions or thick constants stand apart from
    the first row's changes the lists, at creation and with a new table."""
    import types
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    q = u.Quadrupole('q', length=0.3, k1=1.1, slices=4)
    s = u.Sextupole('s', length=0.2, k2=30.0, slices=4)
    v = u.Quadrupole('v', length=0.3, k1=-1.1, slices=4)
    line = u.Line('r', [u.Drift('d', length=0.5), q, u.Drift('e', length=0.4), s, v] * 20)
    prog = C.compile_line(line, 0 if what == 'entry' else u.KICK, where=[])
    table = np.repeat(prog.table, rows, axis=0)
    apart = table.copy()
    for op in prog.ops:
        kind, off = int(op[0]), int(op[2])
        if what == 'entry' and kind == C.OP_THICKQ:
            apart[-1, off] *= 1.0 + 1e-3 * (off % 7)
        if what != 'entry' and kind == C.OP_TEAPOT:
            if what == 'strength':
                apart[-1, off + 5] = 1e-300
            else:  # [A, d, 1/d, A/d] of the inner drift
                apart[-1, off + 2:off + 5] = 5.0, 1 / 5.0, apart[-1, off + 1] / 5.0
    coords = beam(200)
    seed = np.where(np.arange(200) % 2, rows - 1, 0).astype(np.int32)

    def check(dp):
        out = [capi.track(ctx, dp, coords, 3, capi.UFO_MODE_TRACK, f, seed=seed, slots=0)[1:]
               for f in (0, capi.UFO_TRACK_PLAIN)]
        assert same(*out)
        return out[0][1]

    def program(tab):
        return capi.DeviceProgram(ctx, types.SimpleNamespace(ops=prog.ops, table=tab, n_dumps=0))
    dp = program(table)
    first = check(dp)
    dp.set_table(apart)
    second = check(dp)
    assert np.isfinite(first).all() and not np.array_equal(first, second)
    assert np.array_equal(check(program(apart)), second)
    dp.set_table(table)
    assert np.array_equal(check(dp), first)


def test_a_cache_of_many_entries_grows_with_the_launches():
    """A ring of magnets that share no entry: one entry set per magnet and lane, so
    the cache starts small and grows with the launches, past what is kept."""
    import ufo_gb300 as u
    from ufo_gb300 import capi, compiler as C
    ctx = u.context(0)
    rng = np.random.default_rng(6)
    cells = []
    for i in range(120):
        k = 1.0 + 0.01 * rng.standard_normal(2)
        cells += [u.Quadrupole(f'f{i}', length=0.3, k1=k[0]), u.Drift(f'd{i}', length=0.5),
                  u.Quadrupole(f'g{i}', length=0.3, k1=-k[1]), u.Drift(f'e{i}', length=0.5)]
    dp = capi.DeviceProgram(ctx, C.compile_line(u.Line('r', cells), 0, where=[]))
    for n in (40, 300, 2500, 20_000, 70_000, 100_000, 40):
        c = beam(n, n)
        out = [capi.track(ctx, dp, c, 2, capi.UFO_MODE_TRACK, f, slots=0)[1:]
               for f in (0, capi.UFO_TRACK_PLAIN)]
        assert np.isfinite(out[1][1]).all() and same(*out), n
