"""Performance cases: what users of this library have it compute.

Each case is one call (or one forward and backward) of a public entry point on
a ring of this repository: the FODO ring ``c1`` (128 elements), the same with
apertures and multipole errors ``c3`` (144), the light-source ring ``c2`` (1024
elements), that ring with one error seed ``c5``, and the MAD-X storage ring
``alba`` that the tests read (768 elements, combined-function bends with
fringe fields).  ``mode`` is the element model: ``thick`` (the drivers' default:
exact quadrupoles and bends, chromatic), ``kick`` (drift-kick slices in the
reference's operation order), ``fma`` (the same with fused arithmetic) and
``yoshida`` (fourth-order slices, fused).

``exact`` restates the same calls in plain float64 torch operations, from the
element attributes alone.
"""
import copy
import math
import os

import numpy as np
import torch

import ufo_gb300 as u
from ufo_gb300 import diff, workloads

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
COLUMNS = ['x', 'px', 'y', 'py', 'dp']
MODES = {
    'thick': u.DOUBLE_PRECISION,
    'thick32': 0,  # the drivers' default flags: single-precision arrays around FP64 tracking
    'kick': u.KICK | u.DOUBLE_PRECISION,
    'fma': u.KICK | u.FMA | u.DOUBLE_PRECISION,
    'yoshida': u.KICK | u.FMA | u.YOSHIDA | u.DOUBLE_PRECISION,
}
TWISS = ('bx', 'by', 'ax', 'ay', 'dx', 'dpx', 'dy', 'dpy', 'mux', 'muy')


def listed():
    return [
        # linear optics at every element of a ring: what a matching script calls
        # in a loop; three particles, one turn, so latency is all of it
        dict(name='optics_ring', kind='optics', ring='alba', step=1),
        # closed orbits of a ring with misaligned sextupoles (orbit response,
        # error studies): a few hundred dependent one-turn maps, few lanes
        dict(name='orbit_thick', kind='orbit', ring='alba', mode='thick', n=12, iterations=200),
        # Track as constructed by default: 1000 particles, exact thick elements,
        # single-precision arrays
        dict(name='track_default', kind='track', ring='alba', mode='thick32', n=1000, turns=20,
             points=1, every=1),
        # the plain FODO ring, 1024 particles for hundreds of turns (a first script)
        dict(name='track_fodo', kind='track', ring='c1', mode='kick', n=1024, turns=500,
             points=1, every=50),
        # turn-by-turn data at many observation points (beam position monitors):
        # an odd bunch, a large record
        dict(name='track_bpms', kind='track', ring='c2', mode='kick', n=333, turns=40, points=97,
             every=1),
        # a full bunch through the light-source ring in the reference's
        # arithmetic (the parity mode), particles resident to the end
        dict(name='bunch_kick', kind='track', ring='c2', mode='kick', n=65536, turns=32, points=1,
             every=32),
        # the same bunch in fused arithmetic: throughput runs
        dict(name='bunch_fma', kind='track', ring='c2', mode='fma', n=65536, turns=40, points=1,
             every=40),
        # dynamic-aperture scan on a polar grid: most particles are lost early,
        # the survivors decide the time
        dict(name='aperture_fma', kind='aperture', ring='c3', mode='fma', radii=128, angles=128,
             momenta=3, turns=512),
        # a small ragged scan with the default element model (a quick look at a
        # working point)
        dict(name='aperture_thick', kind='aperture', ring='alba', mode='thick', radii=13,
             angles=11, momenta=1, turns=40),
        # error seeds of uneven size in one launch
        dict(name='seeds_fma', kind='seeds', seeds=64, low=64, high=2048, turns_low=64,
             turns_high=256),
        # gradients of closed orbit, tunes and chromaticity by every quadrupole
        # and sextupole strength, forward and backward
        dict(name='optics_gradient', kind='optics_grad', strengths=512),
        # gradient of a bunch's final amplitudes after many turns, checkpointed
        dict(name='amplitude_gradient', kind='amplitude_grad', n=777, turns=32, ck=8),
    ]


def _log(rng, low, high):
    """An integer spread over the logarithm of [low, high]."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


# elements of each ring, and rough costs used only to bound the drawn sizes: one
# element and turn for a lone warp [us], and the element-turns of a full GPU [1/us]
SIZE = {'c1': 128, 'c3': 144, 'c2': 1024, 'c5': 1024, 'alba': 768}
LONE = {'thick': 8.0, 'thick32': 8.0, 'kick': 1.4, 'fma': 0.9, 'yoshida': 2.2}
FULL = {'thick': 1e3, 'thick32': 1e3, 'kick': 1e4, 'fma': 3e4, 'yoshida': 1e4}
BUDGET_US = 2e5


def _turns_for(ring, mode, n):
    """Turns that stay within the largest listed case's time."""
    per_turn = SIZE[ring] * max(LONE[mode], n / FULL[mode])
    return max(1, int(BUDGET_US / per_turn))


def draw(rng):
    kind = rng.choice(['optics', 'orbit', 'track', 'track', 'track', 'aperture', 'aperture',
                       'seeds', 'optics_grad', 'amplitude_grad'])
    if kind == 'optics':
        return dict(kind=kind, ring=rng.choice(['c1', 'alba']), step=_log(rng, 1, 64))
    if kind == 'orbit':
        ring = rng.choice(['c1', 'alba'])
        return dict(kind=kind, ring=ring, mode=rng.choice(['thick', 'kick']), n=_log(rng, 1, 2000),
                    iterations=200 if ring == 'alba' else rng.randint(200, 400))
    if kind == 'track':
        ring = rng.choice(['c1', 'c2', 'c5', 'alba'])
        mode = rng.choice(['thick', 'thick32', 'kick', 'kick', 'fma', 'fma', 'yoshida'])
        if ring == 'c5' and mode in ('thick', 'thick32'):
            mode = 'kick'  # thick elements carry no multipole errors
        n = _log(rng, 1, 65536)
        turns = _log(rng, 1, _turns_for(ring, mode, n))
        points = rng.choice([1, 1, 1, 2, 3, _log(rng, 1, 97)])
        most = max(1, 2_000_000 // (n * points))  # observations kept per particle
        return dict(kind=kind, ring=ring, mode=mode, n=n, turns=turns, points=points,
                    every=min(turns, max(rng.choice([1, 1, 7, turns]), -(-turns // most))))
    if kind == 'aperture':
        mode = rng.choice(['kick', 'fma', 'thick'])
        ring = 'alba' if mode == 'thick' else 'c3'
        momenta = rng.choice([1, 1, 3])
        radii, angles = _log(rng, 3, 160), _log(rng, 3, 128)
        most = _turns_for(ring, mode, 0.3 * radii * angles * momenta)
        return dict(kind=kind, ring=ring, mode=mode, radii=radii, angles=angles, momenta=momenta,
                    turns=_log(rng, min(8, most), min(1024, most)))
    if kind == 'seeds':
        high = _log(rng, 40, 2048)
        low_turns = _log(rng, 8, 128)
        return dict(kind=kind, seeds=_log(rng, 2, 64), low=_log(rng, 8, 40), high=high,
                    turns_low=low_turns, turns_high=low_turns + rng.randint(0, 128))
    if kind == 'optics_grad':
        return dict(kind=kind, strengths=_log(rng, 8, 512))
    turns = _log(rng, 1, 32)
    return dict(kind=kind, n=_log(rng, 1, 777), turns=turns, ck=rng.randint(max(1, -(-turns // 6)), turns))


# ------------------------------------------------------------------ inputs

def _ring(name):
    if name == 'alba':
        return u.Lattice(os.path.join(ROOT, 'tests', 'golden', 'madx', 'alba.mad')).RING
    return getattr(workloads, f'{name}_ring')(u)


def _beam(ring, n, seed):
    """Gaussian bunch [n, 5] (x, px, y, py, dp) with each ring's own sizes."""
    make = workloads.c1_beam if ring == 'c1' else workloads.c2_beam
    return make(n, seed=seed)[:, [0, 1, 2, 3, 5]]


def _points(case, flat):
    """Observation points: the end of the turn, and elements spread over it."""
    k = case['points'] - 1
    return [int(i * len(flat) / k) for i in range(k)] + [-1] if k else [-1]


def _grid(case, seed):
    """Polar amplitude grid [n, 5] at a few momenta; the seed turns the angles
    and stretches the radii a little, so that other seeds are other grids."""
    rng = np.random.default_rng(seed)
    r = np.linspace(0.0, 0.025, case['radii']) * (1 + 0.02 * rng.random())
    t = np.linspace(0.0, math.pi / 2, case['angles']) * (1 - 0.02 * rng.random())
    dps = [0.0] if case['momenta'] == 1 else [-0.02, 0.0, 0.02]
    rr, tt = np.meshgrid(r, t, indexing='ij')
    out = np.zeros((len(dps), rr.size, 5))
    for k, dp in enumerate(dps):
        out[k, :, 0], out[k, :, 2] = (rr * np.cos(tt)).ravel(), (rr * np.sin(tt)).ravel()
        out[k, :, 4] = dp
    return out.reshape(-1, 5)


def _orbit_setup(case, seed):
    """Offsets of a few magnets per orbit: (parameter list, values [n, P])."""
    ring = _ring(case['ring'])
    flat = ring.flatten()
    kind = 'Sextupole' if case['ring'] == 'alba' else 'Quadrupole'
    at = [i for i, e in enumerate(flat) if type(e).__name__ == kind][::7]
    params = [(i, a) for i in at for a in ('dx', 'dy')]
    rng = np.random.default_rng(seed)
    return ring, params, rng.normal(0, 30e-6, (case['n'], len(params)))


def _knobs(ring, seed):
    """Every fifth quadrupole as a matching knob: (flat indices, k1 values)."""
    flat = ring.flatten()
    at = [i for i, e in enumerate(flat) if type(e).__name__ == 'Quadrupole'][::5]
    rng = np.random.default_rng(seed)
    return at, np.array([flat[i].k1 for i in at]) * (1 + 1e-4 * rng.standard_normal(len(at)))


def _seed_setup(case, seed):
    ring = workloads.c1_ring(u)
    rng = np.random.default_rng(case['seeds'])  # the study's sizes; the seed draws its errors
    parts = np.exp(rng.uniform(math.log(case['low']), math.log(case['high']),
                               case['seeds'])).astype(np.int64)
    turns = rng.integers(case['turns_low'], case['turns_high'] + 1, case['seeds'])
    rows = workloads.c4_seed_rows(ring, case['seeds'], seed=seed)
    beam = workloads.c1_beam(int(parts.sum()), seed=seed + 1)
    return ring, workloads.c4_parameters(ring), rows, parts, turns, beam


def _grad_setup(case, seed):
    """The error ring, its quadrupole and sextupole strengths (or an even
    choice of them) a little off the design, and the weights of a scalar
    objective of the eight optics outputs."""
    ring = workloads.c5_ring(u)
    params, vals = workloads.c5_parameters(ring)
    count = case.get('strengths', len(params))
    pick = [j * len(params) // count for j in range(count)]
    params, vals = [params[j] for j in pick], vals[pick]
    rng = np.random.default_rng(seed)
    return ring, params, vals * (1 + 1e-4 * rng.standard_normal(len(vals))), rng.uniform(0.5, 1.5, 8)


def prepare(case, seed):
    kind = case['kind']
    st = {'kind': kind}
    if kind == 'optics':
        ring = _ring(case['ring'])
        at, k1 = _knobs(ring, seed)
        st['sim'] = u.Optics(ring, where=list(range(0, len(ring.flatten()), case['step'])),
                             parameters=[(i, 'k1') for i in at],
                             flags=u.LINEAR | u.ACHROMATIC | u.DOUBLE_PRECISION)
        st['sim'].parameters[0] = k1
    elif kind == 'orbit':
        ring, params, values = _orbit_setup(case, seed)
        st['sim'] = u.ClosedOrbit(ring, flags=MODES[case['mode']], particles=case['n'],
                                  parameters=params, iterations=case['iterations'])
        st['sim'].parameters[:] = values
    elif kind == 'track':
        ring = _ring(case['ring'])
        st['sim'] = u.Track(ring, flags=MODES[case['mode']], turns=case['turns'],
                            particles=case['n'], parameters=COLUMNS, every=case['every'],
                            where=_points(case, ring.flatten()))
        st['sim'].parameters[:] = _beam(case['ring'], case['n'], seed)
    elif kind == 'aperture':
        grid = _grid(case, seed)
        st['sim'] = u.StableAperture(_ring(case['ring']), flags=MODES[case['mode']],
                                     turns=case['turns'], particles=len(grid), parameters=COLUMNS)
        st['sim'].parameters[:] = grid
    elif kind == 'seeds':
        ring, params, rows, parts, turns, beam = _seed_setup(case, seed)
        st['sim'] = u.TrackBatch(ring, params, rows, parts, turns, flags=u.KICK | u.FMA)
        st['sim'].coords[:] = beam
    else:
        ring, params, values, weights = _grad_setup(case, seed)
        st['model'] = diff.OpticsModel(ring, u.KICK, params)
        st['k'] = torch.tensor(values, dtype=torch.float64)
        if kind == 'optics_grad':
            st['weights'] = torch.tensor(weights, dtype=torch.float64)
        else:
            st['beam'] = workloads.c2_beam(case['n'], seed=seed)
            st['turns'], st['ck'] = case['turns'], case['ck']
    return st


def run(state):
    kind = state['kind']
    if kind in ('optics_grad', 'amplitude_grad'):
        k = state['k'].detach().requires_grad_()
        if kind == 'optics_grad':
            out = diff.optics(k, state['model'])
            (out * state['weights']).sum().backward()
        else:
            out = diff.amplitudes(k, state['model'], state['beam'], state['turns'], state['ck'])
            out.sum().backward()
        return {'value': out.detach(), 'grad': k.grad}
    sim = state['sim']
    sim.run()
    if kind == 'optics':
        return {'tunes': np.array([sim.qx, sim.qy]),
                **{a: np.array(getattr(sim, a)) for a in TWISS}}
    if kind == 'orbit':
        return {'orbits': sim.orbits}
    if kind == 'track':
        return {'tracks': sim.tracks, 'lost': sim.lost, 'final': sim.final}
    return {'lost': sim.lost, 'final': sim.final}


# ------------------------------------------------------------------ work

def _flops(e, mode):
    """Floating-point operations of one element's map for one particle: the
    textbook count (a multiply-add is two, a transcendental is one)."""
    t = type(e).__name__
    if t == 'Drift':
        return 4
    if t == 'Aperture':
        return 3
    if t not in ('Quadrupole', 'Sbend', 'Sextupole'):
        return 0
    edges = 7 if t == 'Sbend' and (e.e1 or e.e2) else 0
    if mode.startswith('thick') and t != 'Sextupole':
        return 16 + edges
    top = 2 if t == 'Sextupole' else 1 if e.k1 else 0
    errors = [j for j, v in enumerate(e.dkn) if v] + [j for j, v in enumerate(e.dks) if v]
    top = max([top] + errors)
    kick = 4 if top == 1 else 8 * top + 4 if errors else 10 if top == 2 else 0
    kick += 2 if t == 'Sbend' else 0
    if mode == 'yoshida':
        return e.slices * (4 * 4 + 3 * kick) + edges
    return 4 * (e.slices + 1) + e.slices * kick + edges


def _ring_flops(ring, mode):
    return sum(_flops(e, mode) for e in _ring(ring).flatten())


def work(case):
    kind = case['kind']
    if kind == 'optics':
        n = SIZE[case['ring']] // case['step'] + 1
        return {'bytes': 3 * 48 + n * 10 * 8, 'flops': 3 * _ring_flops(case['ring'], 'thick')}
    if kind == 'orbit':
        # each search step tries one vertex at least
        return {'bytes': 32 * case['n'],
                'flops': case['n'] * case['iterations'] * _ring_flops(case['ring'], case['mode'])}
    if kind == 'track':
        size = 4 if case['mode'] == 'thick32' else 8
        kept = case['turns'] // case['every'] * case['points']
        return {'bytes': case['n'] * size * (5 + 6 * kept + 6) + 4 * case['n'],
                'flops': case['n'] * case['turns'] * _ring_flops(case['ring'], case['mode'])}
    if kind == 'aperture':
        # about three particles in twenty of such a grid live to the end
        n = case['radii'] * case['angles'] * case['momenta']
        return {'bytes': n * (40 + 4 + 48),
                'flops': int(0.15 * n * case['turns'] * _ring_flops(case['ring'], case['mode']))}
    if kind == 'seeds':
        _, _, rows, parts, turns, _ = _seed_setup(case, 0)
        # every magnet carries errors up to order 5 in both lists
        per = sum(4 * (e.slices + 1) + e.slices * 44 + 4 if e.length and type(e).__name__ != 'Drift'
                  else 4 for e in workloads.c1_ring(u).flatten())
        return {'bytes': rows.nbytes + int(parts.sum()) * (48 + 48 + 4),
                'flops': int((parts * turns).sum()) * per}
    per = _ring_flops('c5', 'kick')
    if kind == 'optics_grad':
        # three momenta: a few Newton steps of the map with its four tangent
        # columns, and about twice that backwards
        return {'bytes': case['strengths'] * 16 + 64, 'flops': 3 * 5 * per * (4 + 2)}
    return {'bytes': case['n'] * (48 + 8) + 512 * 16, 'flops': 4 * case['n'] * case['turns'] * per}


# ------------------------------------------------------------------ float64 reference

_W1 = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
YOSHIDA = ((_W1 / 2, _W1), ((1 - _W1) / 2, 1 - 2 * _W1), ((1 - _W1) / 2, _W1), (_W1 / 2, 0.0))


def _series(e, t, linear, k):
    """(normal, skew) multipole strengths k_n of an element, n = 0, 1, ...;
    ``k`` replaces its main strength (a tensor, for derivatives)."""
    main = {'Quadrupole': 1, 'Sbend': 1, 'Sextupole': 2}[t]
    kn, ks = list(e.dkn) + [0.0] * (main + 1 - len(e.dkn)), list(e.dks)
    if k is None:
        k = e.k2 if t == 'Sextupole' else e.k1
    kn[main] = kn[main] + k
    if linear:
        kn, ks = kn[:2], ks[:2]
    ks = ks + [0.0] * (len(kn) - len(ks))
    kn = kn + [0.0] * (len(ks) - len(kn))
    return kn, ks


def _mul(a, b):
    """a * b, with a literal zero left out."""
    return 0.0 if isinstance(a, float) and a == 0.0 else a * b


def _add(a, b):
    if isinstance(a, float) and a == 0.0:
        return b
    return a if isinstance(b, float) and b == 0.0 else a + b


def _kick(s, kn, ks, w, o, h):
    """px -= Re S, py += Im S with S(z) = o w sum (kn + i ks) z^n / n!, and the
    tangent rows s[4..7] where the state carries them."""
    x, px, y, py = s[:4]
    sr = si = dr = di = 0.0
    for n in range(len(kn) - 1, -1, -1):
        f = w / math.factorial(n)
        if len(s) > 4:
            dr, di = (_add(_add(_mul(dr, x), _mul(di, -y)), sr),
                      _add(_add(_mul(dr, y), _mul(di, x)), si))
        sr, si = (_add(_add(_mul(sr, x), _mul(si, -y)), _mul(kn[n], f)),
                  _add(_add(_mul(sr, y), _mul(si, x)), _mul(ks[n], f)))
    out = [x, _add(_add(px, _mul(sr, -o)), _mul(h, -x)), y, _add(py, _mul(si, o))]
    if len(s) > 4:
        dr, di = (v * o if torch.is_tensor(v) else torch.full_like(x, v) * o for v in (dr, di))
        X, PX, Y, PY = s[4:]
        out += [X, PX - (dr + h)[:, None] * X + di[:, None] * Y, Y,
                PY + di[:, None] * X + dr[:, None] * Y]
    return out


def _drift(s, L):
    out = [s[0] + s[1] * L, s[1], s[2] + s[3] * L, s[3]]
    if len(s) > 4:
        out += [s[4] + s[5] * L, s[5], s[6] + s[7] * L, s[7]]
    return out


def _edge(s, e, angle, o):
    curv = e.angle / e.length * o
    fringe = e.hgap * e.fint
    psi = angle - 2 * curv * fringe / math.cos(angle) * (1 + math.sin(angle) ** 2)
    tpsi = torch.tan(psi) if torch.is_tensor(psi) else math.tan(psi)
    return [s[0], s[1] + s[0] * curv * math.tan(angle), s[2], s[3] - s[2] * curv * tpsi]


def _plane(q, p, K, L, disp):
    """One plane of a thick element: q'' = -K q + disp."""
    K = K if torch.is_tensor(K) else torch.full_like(q, K)
    w = torch.sqrt(torch.abs(K))
    foc = K > 0
    C = torch.where(foc, torch.cos(w * L), torch.cosh(w * L))
    S = torch.where(foc, torch.sin(w * L), torch.sinh(w * L))
    free = w == 0
    w1 = torch.where(free, torch.ones_like(w), w)
    sw = torch.where(free, torch.full_like(w, L), S / w1)
    d1 = torch.where(free, torch.zeros_like(w),
                     torch.where(foc, 1 - C, C - 1) / (w1 * w1))
    return (q * C + p * sw + disp * d1,
            torch.where(foc, -S, S) * w * q + C * p + disp * torch.where(free, w, sw))


def _element(s, e, mode, o, dp, linear=False, achro=False, shift=None, k=None):
    """One element's map on s = [x, px, y, py] (tensors over particles)."""
    t = type(e).__name__
    if t == 'Drift':
        return _drift(s, e.length)
    if t == 'Aperture':
        out = s[0] ** 2 + s[2] ** 2 < 1e-4
        return [torch.where(out, s[0], torch.full_like(s[0], math.nan))] + list(s[1:])
    if t not in ('Quadrupole', 'Sbend', 'Sextupole'):
        return s
    ok = 1.0 if achro else o
    dx, dy = (e.dx, e.dy) if shift is None else shift
    s = [s[0] - dx, s[1], s[2] - dy] + list(s[3:])
    bend = t == 'Sbend'
    if bend and (e.e1 or e.e2):
        s = _edge(s, e, e.e1, ok)
    if mode.startswith('thick') and t != 'Sextupole':
        h = e.angle / e.length if bend else 0.0
        Kx, Ky = (e.k1 + h * h) * ok, -e.k1 * ok
        x, px = _plane(s[0], s[1], Kx, e.length, dp * h * ok)
        y, py = _plane(s[2], s[3], Ky, e.length, 0.0)
        s = [x, px, y, py]
    else:
        N, L = e.slices, e.length
        kn, ks = _series(e, t, linear, k)
        weak = e.angle ** 2 / (N * L) if bend else 0.0
        if mode == 'yoshida':
            for _ in range(N):
                for c, d in YOSHIDA:
                    s = _drift(s, c * L / N)
                    if d:
                        s = _kick(s, kn, ks, L / N * d, ok, weak * d)
        else:
            outer = L / 2 if N == 1 else L / (2 * (1 + N))
            inner = (L - 2 * outer) / (N - 1) if N > 1 else 0.0
            s = _drift(s, outer)
            for i in range(N):
                s = _kick(s, kn, ks, L / N, ok, weak)
                s = _drift(s, inner if i < N - 1 else outer)
    if bend and (e.e1 or e.e2):
        s = _edge(s, e, e.e2, ok)
    return [s[0] + dx, s[1], s[2] + dy] + list(s[3:])


def _operations(flat, mode):
    """Rough number of tensor operations of one turn."""
    n = 0
    for e in flat:
        t = type(e).__name__
        if t in ('Quadrupole', 'Sbend', 'Sextupole'):
            errors = len(e.dkn) + len(e.dks) > 0
            kick = 2 + 8 * len(e.dkn) if errors else 16 if t == 'Sextupole' else 8
            n += 60 if mode.startswith('thick') and t != 'Sextupole' else \
                e.slices * (4 + kick) * (4 if mode == 'yoshida' else 1)
        else:
            n += 4
    return n


MOST_OPERATIONS = 1_800_000  # tensor operations that take some ten seconds


def _device():
    return 'cuda' if torch.cuda.is_available() else 'cpu'


def _exact_track(ring, mode, coords, turns, where, every, pturns=None, shifts=None, series=None):
    """Tracks [n, slots, 6] and final coordinates [n, 6] in float64, or None
    where it would take too long."""
    flat = ring.flatten()
    if turns * _operations(flat, mode) > MOST_OPERATIONS:
        return None
    dev = _device()
    z0 = torch.tensor(coords, dtype=torch.float64, device=dev)
    s, dp = [z0[:, j] for j in range(4)], z0[:, 5]
    o = 1.0 / (1.0 + dp)
    alive = torch.ones_like(dp, dtype=torch.bool)
    rows = []
    dumps = sorted(p for p in where if p >= 0)

    def record(now):
        rows.append(torch.stack(list(now) + [z0[:, 4], dp], dim=1).masked_fill(~alive[:, None], 0))

    for t in range(turns):
        if pturns is not None:
            alive = alive & (t < pturns)
        now = s
        seen = (t + 1) % every == 0
        for i, e in enumerate(flat):
            if seen and i in dumps:
                record(now)
            if series is not None and i in series:
                e = series[i]
            now = _element(now, e, mode, o, dp, shift=None if shifts is None else shifts.get(i))
        if seen and -1 in where:
            record(now)
        s = [torch.where(alive, a, b) for a, b in zip(now, s)]
        alive = alive & ~torch.isnan(s[0])
    final = torch.stack(s + [z0[:, 4], dp], dim=1)
    tracks = torch.stack(rows, dim=1) if rows else None
    return (None if tracks is None else tracks.cpu().numpy()), final.cpu().numpy()


class _Magnet:
    """An element with per-particle error strengths in place of its lists."""

    def __init__(self, e, dkn, dks):
        self.__dict__.update(e.__dict__)
        self.dkn, self.dks = dkn, dks


def _named(e, dkn, dks):
    return type(type(e).__name__, (_Magnet,), {})(e, dkn, dks)


def _closed_orbits(ring, mode, dps, shifts=None, strengths=None, steps=12):
    """Fixed points of the one-turn map at each dp, with the one-turn matrix
    there: Newton on the map and its central differences."""
    flat = ring.flatten()
    dev = 'cpu'
    dp = torch.as_tensor(dps, dtype=torch.float64, device=dev)
    n = len(dp)

    def turn(z):
        m = len(z) // n
        d = dp.repeat(m)
        o = 1.0 / (1.0 + d)
        s = [z[:, j] for j in range(4)]
        for i, e in enumerate(flat):
            shift = None if shifts is None or i not in shifts else \
                tuple(v.repeat(m) for v in shifts[i])
            s = _element(s, e, mode, o, d, shift=shift,
                         k=None if strengths is None else strengths.get(i))
        return torch.stack(s, dim=1)

    h = 1e-6
    z = torch.zeros((n, 4), dtype=torch.float64)
    for _ in range(steps):
        probe = [z] + [z + sign * h * torch.eye(4, dtype=torch.float64)[j]
                       for j in range(4) for sign in (1, -1)]
        f = turn(torch.cat(probe)).reshape(9, n, 4)
        J = torch.stack([(f[1 + 2 * j] - f[2 + 2 * j]) / (2 * h) for j in range(4)], dim=2)
        step = torch.linalg.solve(J - torch.eye(4, dtype=torch.float64), z - f[0])
        z = z + step
        if float(step.abs().max()) < 1e-16:
            break
    return z


def _exact_optics(case, seed):
    ring = _ring(case['ring'])
    flat = ring.flatten()
    for i, k1 in zip(*_knobs(ring, seed)):
        flat[i] = copy.copy(flat[i])
        flat[i].k1 = k1
    z = torch.zeros((3, 6), dtype=torch.float64)
    z[0, 0] = z[0, 2] = z[1, 1] = z[1, 3] = z[2, 5] = 1.0
    s, dp = [z[:, j] for j in range(4)], z[:, 5]
    one = torch.ones_like(dp)
    rows = []
    for i, e in enumerate(flat):
        if i % case['step'] == 0:
            rows.append(torch.stack(s, dim=1))
        s = _element(s, e, 'thick', one, dp, linear=True, achro=True)
    rows.append(torch.stack(s, dim=1))
    r = torch.stack(rows).numpy()  # [points, 3 columns, 4]
    out = {a: np.empty(len(r)) for a in TWISS}
    tunes = np.empty(2)
    for plane, q in ((0, 0), (1, 2)):
        R11, R21 = r[:, 0, q], r[:, 0, q + 1]
        R12, R22 = r[:, 1, q], r[:, 1, q + 1]
        d, dpr = r[:, 2, q], r[:, 2, q + 1]
        c = 0.5 * (R11[-1] + R22[-1])
        if abs(c) > 1:
            return None
        sn = math.copysign(math.sqrt(1 - c * c), R12[-1])
        b0, a0 = R12[-1] / sn, 0.5 * (R11[-1] - R22[-1]) / sn
        g0 = (1 + a0 * a0) / b0
        tunes[plane] = math.atan2(sn, c) % (2 * math.pi) / (2 * math.pi)
        p = 'xy'[plane]
        out['b' + p] = R11 * R11 * b0 - 2 * R11 * R12 * a0 + R12 * R12 * g0
        out['a' + p] = -(R11 * R21 * b0 - (R11 * R22 + R12 * R21) * a0 + R12 * R22 * g0)
        out['mu' + p] = np.arctan2(R12, b0 * R11 - a0 * R12)
        if plane == 0:  # periodic horizontal dispersion; the vertical one starts at 0
            M = np.array([[R11[-1], R12[-1]], [R21[-1], R22[-1]]])
            eta = np.linalg.solve(np.eye(2) - M, np.array([d[-1], dpr[-1]]))
        else:
            eta = np.zeros(2)
        out['d' + p] = R11 * eta[0] + R12 * eta[1] + d
        out['dp' + p] = R21 * eta[0] + R22 * eta[1] + dpr
    return {'tunes': tunes, **out}


def _tangent_turn(flat, z, dp, k, slots):
    """One turn of the kick model with its 4x4 tangent, differentiable in the
    strengths ``k`` (element index -> entry of k)."""
    eye = torch.eye(4, dtype=torch.float64).expand(len(z), 4, 4)
    s = [z[:, j] for j in range(4)] + [eye[:, j] for j in range(4)]
    o = 1.0 / (1.0 + dp)
    for i, e in enumerate(flat):
        s = _element(s, e, 'kick', o, dp, k=k[slots[i]] if i in slots else None)
    return torch.stack(s[:4], dim=1), torch.stack(s[4:], dim=1)


def _exact_optics_grad(case, seed):
    ring, params, values, weights = _grad_setup(case, seed)
    flat = ring.flatten()
    slots = {i: j for j, (i, _) in enumerate(params)}
    h = 1e-4
    dps = torch.tensor([0.0, h, -h], dtype=torch.float64)
    fixed = {i: float(values[j]) for i, j in slots.items()}
    z = _closed_orbits(ring, 'kick', dps, strengths=fixed)
    k = torch.tensor(values, dtype=torch.float64, requires_grad=True)
    # one more Newton step with the map's dependence on k: the fixed point and
    # its first derivative
    F, M = _tangent_turn(flat, z, dps, k, slots)
    J = M.detach()
    z = z - torch.linalg.solve(J - torch.eye(4, dtype=torch.float64), F - z)
    _, M = _tangent_turn(flat, z, dps, k, slots)
    q = []
    for a in (0, 2):
        c = 0.5 * (M[:, a, a] + M[:, a + 1, a + 1])
        sn = torch.sqrt(1 - c * c) * torch.sign(M[:, a, a + 1].detach())
        mu = torch.atan2(sn, c)
        q.append(torch.where(mu < 0, mu + 2 * math.pi, mu) / (2 * math.pi))
    q = torch.stack(q, dim=1)
    out = torch.cat([z[0], q[0], (q[1] - q[2]) / (2 * h)])
    (out * torch.tensor(weights, dtype=torch.float64)).sum().backward()
    return {'value': out.detach().numpy(), 'grad': k.grad.numpy()}


def _exact_amplitude_grad(case, seed):
    ring, params, values, _ = _grad_setup(case, seed)
    flat = ring.flatten()
    # the graph of every operation is kept: memory and time bound the turns
    if case['turns'] * _operations(flat, 'kick') > MOST_OPERATIONS // 4:
        return None
    slots = {i: j for j, (i, _) in enumerate(params)}
    k = torch.tensor(values, dtype=torch.float64, requires_grad=True, device=_device())
    beam = torch.tensor(workloads.c2_beam(case['n'], seed=seed), device=_device())
    s, dp = [beam[:, j] for j in range(4)], beam[:, 5]
    o = 1.0 / (1.0 + dp)
    strengths = k.unbind()
    for _ in range(case['turns']):
        for i, e in enumerate(flat):
            s = _element(s, e, 'kick', o, dp, k=strengths[slots[i]] if i in slots else None)
    amp = s[0] ** 2 + s[2] ** 2
    amp.sum().backward()
    return {'value': amp.detach().cpu().numpy(), 'grad': k.grad.cpu().numpy()}


def exact(case, seed):
    kind = case['kind']
    if kind == 'optics':
        return _exact_optics(case, seed)
    if kind == 'orbit':
        ring, params, values = _orbit_setup(case, seed)
        if 9 * 6 * _operations(ring.flatten(), case['mode']) * max(1, case['n'] / 200) > \
                MOST_OPERATIONS:
            return None
        v = torch.tensor(values, dtype=torch.float64)
        shifts = {i: (v[:, 2 * j], v[:, 2 * j + 1])
                  for j, i in enumerate(dict.fromkeys(i for i, _ in params))}
        z = _closed_orbits(ring, case['mode'], np.zeros(case['n']), shifts=shifts)
        return {'orbits': z.numpy()}
    if kind == 'aperture':
        return None  # loss turns are counts, and a lost particle's last state is chaotic
    if kind == 'track':
        ring = _ring(case['ring'])
        pool = _beam(case['ring'], case['n'], seed)
        if case['mode'] == 'thick32':
            pool = pool.astype(np.float32).astype(np.float64)
        coords = np.zeros((len(pool), 6))
        coords[:, [0, 1, 2, 3, 5]] = pool
        got = _exact_track(ring, case['mode'], coords, case['turns'],
                           _points(case, ring.flatten()), case['every'])
        if got is None:
            return None
        return {'tracks': got[0], 'lost': None, 'final': got[1]}
    if kind == 'seeds':
        ring, params, rows, parts, turns, beam = _seed_setup(case, seed)
        flat = ring.flatten()
        if int(turns.max()) * 128 * 120 > MOST_OPERATIONS:
            return None
        dev = _device()
        per = torch.tensor(np.repeat(rows, parts, axis=0), device=dev)
        shifts, series = {}, {}
        for i in dict.fromkeys(i for i, _ in params):
            cols = {a: per[:, j] for j, (m, a) in enumerate(params) if m == i}
            shifts[i] = (cols['dx'], cols['dy'])
            zero = [0.0, 0.0]
            series[i] = _named(flat[i], zero + [cols[f'dk{j}'] for j in range(2, 6)],
                               zero + [cols[f'dk{j}s'] for j in range(2, 6)])
        pt = torch.tensor(np.repeat(turns, parts), device=dev)
        got = _exact_track(ring, 'kick', beam, int(turns.max()), [], 1, pturns=pt,
                           shifts=shifts, series=series)
        return None if got is None else {'lost': None, 'final': got[1]}
    if kind == 'optics_grad':
        return _exact_optics_grad(case, seed)
    return _exact_amplitude_grad(case, seed)
