"""The eight-lane tangent and adjoint kernels against the job-per-lane ones,
which batches beyond 32 jobs per SM take."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _line(name):
    import os
    import ufo_gb300 as u
    if name == 'alba':
        return u.Lattice(os.path.join(H.HERE, 'golden', 'madx', 'alba.mad')).RING, 0
    err = dict(dkn=[0, 0, 3.0, 50.0, 2e3], dks=[1e-5, 1e-3, 1.0, 0, 4e3, 1e5])
    return u.Line('r', [
        u.Quadrupole('a', length=0.3, k1=1.1, slices=4, dx=1e-4, dy=-1e-4, **err),
        u.Drift('d', length=0.7), u.Sextupole('s', length=0.2, k2=30.0, slices=3),
        u.Sbend('b', length=1.1, angle=0.1, k1=-0.3, e1=0.02, e2=0.01, slices=8),
        u.Quadrupole('c', length=0.25, k1=-1.0, slices=11),
        u.Multipole('m', knl=[0, 0.05, 2.0], ksl=[1e-5]),
        u.Sextupole('t', length=0.15, k2=-40.0, slices=1)]), u.KICK


@pytest.mark.parametrize('name', ['mixed', 'alba'])
@pytest.mark.parametrize('jobs', [1, 4, 37])
def test_eight_lanes_match_one_lane(name, jobs):
    """Final state, tangent, start-state cotangent and parameter cotangents of
    the first jobs of a large batch and of the same jobs alone (seeds too).
    Both run the same operations except for the sums of products that a
    parameter's cotangent collects, so states are equal and cotangents agree to
    the rounding of some thousand terms: 1e3 eps of the largest."""
    import torch
    import ufo_gb300 as u
    from ufo_gb300 import diff as D
    line, flags = _line(name)
    flat = line.flatten()
    params = [(i, 'k1') for i, e in enumerate(flat) if type(e).__name__ in ('Quadrupole', 'Sbend')]
    params += [(i, 'k2') for i, e in enumerate(flat) if type(e).__name__ == 'Sextupole']
    base = np.array([getattr(flat[i], a) for i, a in params])
    rows = base * (1 + 1e-3 * np.arange(3)[:, None])
    eng = D.DiffEngine(D.DiffProgram(line, flags, params, rows))
    many = 32 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    rng = np.random.default_rng(jobs)
    z = rng.normal(0, 1e-4, (many, 4))
    o = 1 / (1 + rng.normal(0, 1e-3, many))
    seed = (np.arange(many) % 3).astype(np.int32)
    zb, tb = rng.normal(0, 1, (many, 4)), rng.normal(0, 1, (many, 16))
    turns, ck = (3, 2) if name == 'mixed' else (1, 1)
    got = []
    for n in (many, jobs):
        out, st = eng.forward(z[:n], o[:n], turns, tangent=True, ck=ck, seed=seed[:n])
        zbar, pbar = eng.reverse(st, zb[:n], tb[:n])
        got.append((out[:jobs], zbar[:jobs], pbar[:jobs]))
    (o1, z1, p1), (o8, z8, p8) = got
    assert np.array_equal(o1, o8)
    eps = np.finfo(float).eps
    assert np.max(np.abs(z8 - z1)) <= 1e3 * eps * np.max(np.abs(z1))
    assert np.max(np.abs(p8 - p1)) <= 1e3 * eps * np.max(np.abs(p1))
