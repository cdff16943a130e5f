"""The two-lane kernel's opcode lists and launch plans on the CPU: what the
kernel is going to walk stays within the coefficient cache and the table."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import helpers as H

OP_DRIFT, OP_KICK, OP_TEAPOT, OP_ALIGN, OP_EDGE, OP_THICKQ, OP_THICKB = 1, 2, 3, 4, 5, 6, 7
OP_APERTURE, OP_OBSERVE, OP_DYNKICK = 9, 10, 11
PV_SEGMENT, PV_EDGE_PSI, PV_THICKQ, PV_THICKB, PV_OBSERVE, PV_WIDE = 0, 6, 7, 8, 10, 12
PF_FILL = 1 << 24
CACHED = {PV_THICKQ: 5, PV_THICKB: 7, PV_EDGE_PSI: 1}  # fields of the coefficient cache


@pytest.fixture(scope='module')
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp('pair') / 'pair_list_host.so')
    subprocess.run(['g++', '-std=c++17', '-O1', '-shared', '-fPIC', '-o', so,
                    os.path.join(H.HERE, 'pair_list_host.cpp')], check=True)
    return ctypes.CDLL(so)


def decode(host, ops, table, most=2 ** 31 - 1):
    """(strict list, FMA list, cache fields) of an opcode list and table."""
    ops = np.ascontiguousarray(ops, np.int32).reshape(-1, 8)
    table = np.ascontiguousarray(np.atleast_2d(table), np.float64)
    out = np.zeros((8 * len(ops) + 64, 4), np.int32)
    info = np.zeros(8, np.int64)
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (ops, table, out, info)]
    rc = host.pair_lists(p[0], len(ops), p[1], ctypes.c_int64(table.shape[1]), len(table),
                         ctypes.c_int(most), p[2], ctypes.c_int64(out.size), p[3])
    assert rc == 0 and info[0] == 1
    out = out[:info[1]]
    lists = []
    for part, wide in ((out[:info[2]], info[6]), (out[info[2]:], info[7])):
        part = part[:2 * len(ops) + 4]  # without the cache-filling ops
        end = next(i for i, w in enumerate(part)
                   if w[0] & 0xff == PV_SEGMENT and w[3] <= w[2])
        lists.append(part[:end])
        assert wide == sum((h & 0xff) == PV_WIDE for h in lists[-1][:, 0])
    return lists[0], lists[1], int(info[3])


def walk(lst, fields, stride, n_ops):
    """Every entry reads constants of the row and, if cached, fields of the
    cache; an op run by the one-lane code has its segment to itself; the
    segments cover the opcode list."""
    at, alone = 0, None
    for head, toff, a, b in lst.tolist():
        v = head & 0xff
        assert 0 <= toff < stride
        if v == PV_SEGMENT:
            assert a == at and b > a
            at, alone, count = b, None, 0
            continue
        count += 1
        assert alone is None and (v != PV_WIDE or count == 1)
        if v == PV_WIDE:
            alone = True
        if v in CACHED:
            assert 0 <= a and a + CACHED[v] <= fields
    assert at == n_ops


def thick_quads(k1):
    """A list of thick quadrupoles (constants k1, length), one row per row of k1."""
    k1 = np.atleast_2d(k1)
    n = k1.shape[1]
    ops = [[OP_THICKQ, 0, 2 * i, 0, 0, 0, 0, 0] for i in range(n)]
    table = np.zeros((len(k1), 2 * n))
    table[:, 0::2], table[:, 1::2] = k1, 0.3
    return ops, table


def test_thick_elements_without_room_in_the_cache_run_one_lane(host):
    """A captured launch keeps the cache's size.  Elements that shared an entry
    and no longer do have none: they go through the one-lane code instead of
    reading an entry that is not there."""
    ops, table = thick_quads([[1.1] * 4] * 3)
    strict, fma, fields = decode(host, ops, table)
    assert fields == 5
    apart = table.copy()
    apart[1, 4] = 1.2  # the third quadrupole differs in one row
    strict, fma, again = decode(host, ops, apart, most=fields)
    assert again == fields
    for lst in (strict, fma):
        walk(lst, fields, table.shape[1], len(ops))
        kinds = [h & 0xff for h in lst[:, 0]]
        assert kinds.count(PV_THICKQ) == 3 and kinds.count(PV_WIDE) == 1
        assert sum(bool(h & PF_FILL) for h in lst[:, 0]) == 1
    # bends and fringe edges take what is left, or nothing
    ops = [[OP_THICKQ, 0, 0, 0, 0, 0, 0, 0], [OP_THICKB, 0, 2, 0, 0, 0, 0, 0],
           [OP_EDGE, 1 << 3 | 1 << 5, 5, 0, 0, 0, 0, 0], [OP_EDGE, 1 << 3 | 1 << 5, 11, 0, 0, 0, 0, 0]]
    table = np.linspace(0.1, 1.0, 17)
    for most in range(16):
        strict, _, fields = decode(host, ops, table, most)
        assert fields <= most
        walk(strict, fields, 17, 4)


def slices(host, n, turns, n_ops, sms=152):
    out = np.zeros(4, np.int64)
    host.pair_slices(ctypes.c_int64(n), turns, n_ops, sms, 16, ctypes.c_int64(sms * 512),
                     out.ctypes.data_as(ctypes.c_void_p))
    return out.tolist()


@pytest.mark.parametrize('n_ops', [0, 1, 16, 128, 8192, 1_000_000])
@pytest.mark.parametrize('turns', [1, 2, 3, 1000, 2 ** 30, 2 ** 31 - 2, 2 ** 31 - 1])
def test_slices_cover_every_turn_count(host, turns, n_ops):
    """Every slice but the last is whole and the last is not empty, up to the
    turn counts that stand for "until all are lost"."""
    for n in (1, 152 * 8 * 16, 152 * 8 * 16 + 17, 38_912, 65_536):
        groups, count, q, warps = slices(host, n, turns, n_ops)
        if not groups:
            continue
        assert turns >= 2 and groups == (n + 15) // 16 and warps in (8, 12, 16)
        assert count >= 1 and q >= 1 and (count - 1) * q < turns <= count * q
        assert groups * count < 2 ** 63


def test_slices_end_where_whole_runs_refill_their_lanes(host):
    """Up to 32 groups of 16 per SM."""
    assert slices(host, 152 * 32 * 16, 1000, 128)[0] == 152 * 32
    assert slices(host, 152 * 32 * 16 + 1, 1000, 128)[0] == 0
    assert slices(host, 152 * 8 * 16, 1000, 128)[0] == 0
    assert slices(host, 152 * 8 * 16 + 1, 1000, 128)[0] == 152 * 8 + 1


def test_ops_without_constants_read_none(host):
    """The kernel loads the first constant of the op ahead: an op that has none may
    stand at the end of the row (offset = stride), where there is none to load."""
    for kind, words in ((0, [0] * 5), (OP_OBSERVE, [0] * 5), (OP_APERTURE, [0] * 5),
                        (OP_DYNKICK, [0] * 5), (OP_KICK, [1, 1, 0, 0, 0])):
        ops = [[OP_DRIFT, 0, 0, 0, 0, 0, 0, 0], [kind, 0, 1, *words], [OP_DRIFT, 0, 0, 0, 0, 0, 0, 0]]
        strict, fma, fields = decode(host, ops, [0.5])
        for lst in (strict, fma):
            walk(lst, fields, 1, 3)
            assert sum((h & 0xff) == PV_OBSERVE for h in lst[:, 0]) == (kind == OP_OBSERVE)


def use(host, n, ops=200, wide=0, thick=False, general=False, fma=False, uneven=False, scan=False,
        row=1000):
    return bool(host.pair_use(ops, wide, int(thick), int(general), ctypes.c_int64(n), 152, int(fma),
                              int(uneven), int(scan), ctypes.c_int64(row)))


@pytest.mark.parametrize('fma', [False, True])
@pytest.mark.parametrize('general', [False, True])
def test_ops_without_a_two_lane_form_bound_the_two_lane_kernel(host, general, fma):
    """The larger the launch, the fewer of them; without any the sizes alone decide."""
    sizes = (1, 1000, 152 * 5 * 16, 152 * 8 * 16, 152 * 9 * 16, 65_536, 1_000_000)
    for extra in ({}, {'uneven': True}, {'scan': True}):
        most = []
        for n in sizes:
            took = [use(host, n, 400, w, general=general, fma=fma, **extra) for w in range(401)]
            assert took == sorted(took, reverse=True)  # no more once there are too many
            most.append(sum(took))
        assert all(a >= b for a, b in zip(most, most[1:]))
        assert 40 <= most[0] <= 81 and most[-1] <= 13
    assert use(host, 10 ** 6) and not use(host, 10 ** 6, fma=True)
    for n in sizes:  # thick rings: up to a quarter, then a fifth at any size
        most = 50 if n <= 152 * 8 * 16 else 40
        assert use(host, n, 200, most, thick=True) and not use(host, n, 200, most + 1, thick=True)


def test_uneven_fused_launches_end_where_whole_warps_win(host):
    """General magnets, particles with their own turn counts: the two-lane kernel
    up to 44 warps per SM (107,008 particles), strict at any size."""
    n = 152 * 44 * 16
    assert use(host, n, general=True, fma=True, uneven=True)
    assert not use(host, n + 1, general=True, fma=True, uneven=True)
    assert not use(host, 1_145_971, general=True, fma=True, uneven=True)
    assert use(host, 1_145_971, general=True, uneven=True)
    assert use(host, 1_145_971, general=True, fma=True, scan=True)


def test_scans_refill_from_a_queue_only_where_it_is_long(host):
    """Untuned scans: all resident up to 10 warps per SM, then 8; tuned launches
    and plain tracking get what they ask for, at most 16."""
    def warps(n, tuning=16, scan=False):
        return host.pair_resident(ctypes.c_int64(n), 152, tuning, int(scan))
    full = 152 * 10 * 16
    assert [warps(n, scan=True) for n in (1, full, full + 1, 10 ** 7)] == [16, 16, 8, 8]
    for n in (1, full, 10 ** 7):
        assert [warps(n, t) for t in (1, 3, 7, 8, 15, 16, 32)] == [2, 6, 14, 16, 16, 16, 16]


def test_fused_launches_of_general_magnets_end_where_their_rows_leave_l1(host):
    for row, most in ((0, 13), (65_536, 13), (65_537, 11), (10 ** 9, 11)):
        n = 152 * most * 16
        assert use(host, n, general=True, fma=True, row=row)
        assert not use(host, n + 1, general=True, fma=True, row=row)
        assert use(host, 152 * 12 * 16, general=True, row=row)
        assert not use(host, 152 * 12 * 16 + 1, general=True, row=row)
