"""Edges of the differentiation kernels' inputs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def forward(ops, tab, z0, tangent, n_ops=None, turns=1):
    """ufo_diff_forward on device buffers; ``ops`` a device tensor."""
    import torch
    from ufo_gb300 import capi
    dev = torch.device('cuda', 0)
    n = len(z0)
    tab = torch.as_tensor(np.atleast_2d(tab), device=dev)
    z = torch.as_tensor(np.ascontiguousarray(z0, np.float64), device=dev)
    o = torch.ones(n, dtype=torch.float64, device=dev)
    out = torch.zeros((n, 20), dtype=torch.float64, device=dev)
    rc = capi.load().ufo_diff_forward(
        capi.ptr(ops.data_ptr()), ops.numel() // 8 if n_ops is None else n_ops,
        capi.ptr(tab.data_ptr()), ctypes.c_int64(tab.shape[1]), None, 0, 0, n,
        capi.ptr(z.data_ptr()), capi.ptr(o.data_ptr()), turns, turns, int(tangent), None,
        capi.ptr(out.data_ptr()), capi.ptr(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize('tangent', [False, True])
def test_an_empty_opcode_list_is_the_identity(tangent):
    import torch
    z0 = np.arange(20.0).reshape(5, 4)
    ops = torch.zeros(8, dtype=torch.int32, device='cuda:0')
    out = forward(ops, np.zeros(1), z0, tangent, n_ops=0, turns=3)
    assert np.array_equal(out[:, :4], z0)
    if tangent:
        assert np.array_equal(out[:, 4:], np.tile(np.eye(4).ravel(), (5, 1)))


@pytest.mark.parametrize('tangent', [False, True])
def test_the_opcode_list_needs_no_more_than_int_alignment(tangent):
    """A list that starts 4, 8 or 12 bytes off a 16-byte boundary, as a slice of a
    caller's array may."""
    import torch
    D_DRIFT, D_ALIGN = 1, 4
    words = [[D_DRIFT, 0, 0, 0, 0, -1, 0, 0], [D_ALIGN, 0, 1, 0, 0, -1, 0, 0],
             [D_DRIFT, 0, 3, 0, 0, -1, 0, 0]]
    tab = [0.5, 1e-3, -2e-3, 0.25]
    z0 = np.arange(28.0).reshape(7, 4)
    want = z0.copy()
    want[:, 0::2] = (z0[:, 0::2] + 0.5 * z0[:, 1::2] - np.array(tab[1:3])) + 0.25 * z0[:, 1::2]
    for off in range(4):
        store = torch.zeros(24 + off, dtype=torch.int32, device='cuda:0')
        store[off:] = torch.tensor(words, dtype=torch.int32).flatten().to(store.device)
        ops = store[off:]
        assert ops.data_ptr() % 16 == 4 * off
        out = forward(ops, tab, z0, tangent)
        assert np.allclose(out[:, :4], want, rtol=1e-15, atol=1e-15)


@pytest.mark.parametrize('tangent', [False, True])
def test_weak_focusing_leaves_the_vertical_plane_alone(tangent):
    """A bend's weak focusing acts on x; an infinite y keeps its finite slope."""
    import ufo_gb300 as u
    from ufo_gb300 import diff
    line = u.Line('l', [u.Sbend('b', length=1.0, angle=0.1, slices=3), u.Drift('d', length=0.5)])
    eng = diff.DiffEngine(diff.DiffProgram(line, u.KICK, []))
    z0 = np.array([[1e-3, 1e-4, np.inf, 2e-4], [1e-3, 1e-4, -1e-3, 2e-4]])
    out, _ = eng.forward(z0, np.ones(2), 2, tangent=tangent)
    assert np.array_equal(out[0, :2], out[1, :2]) and out[0, 2] == np.inf
    assert out[0, 3] == out[1, 3] == 2e-4


@pytest.mark.parametrize('tangent', [False, True])
def test_a_teapot_without_slices_is_its_outer_drift_both_ways(tangent):
    import types
    from ufo_gb300 import diff
    D_TEAPOT = 2
    prog = types.SimpleNamespace(
        ops=np.array([[D_TEAPOT, 0, 0, 0, 1, -1, 0, 0]], np.int32),
        tab=np.array([[0.5, 0.1, 0.0, 0.0, 0.0, 0.25, 0.0, 0.0]]), n_seeds=1, tab_stride=8,
        kicks_per_turn=0, n_params=0)
    eng = diff.DiffEngine(prog)
    z0 = np.arange(12.0).reshape(3, 4)
    out, state = eng.forward(z0, np.ones(3), 1, tangent=tangent)
    want = z0.copy()
    want[:, 0::2] += 0.5 * z0[:, 1::2]
    assert np.array_equal(out[:, :4], want)
    zbar = np.arange(12.0)[::-1].reshape(3, 4).copy()
    got, _ = eng.reverse(state, zbar, np.zeros((3, 16)) if tangent else None)
    want = zbar.copy()
    want[:, 1::2] += 0.5 * zbar[:, 0::2]
    assert np.array_equal(got, want)
