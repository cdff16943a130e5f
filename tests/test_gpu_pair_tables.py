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
