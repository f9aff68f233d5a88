"""The point sort (gale_b200/csrc/gg_points.cu; needs a B200) where its paths change: element
counts around the register networks (16, 32, 64), above them, and more points than one
window of the scatter.  Order and offsets are those of a stable sort by element."""
import ctypes as C
import time

import numpy as np
import pytest

from gale_b200 import abi
from gale_b200.stokes import GaleError, Mesh, StokesProblem

pytestmark = pytest.mark.gpu


def noalloc(mesh, x, nel):
    torch = pytest.importorskip("torch")
    n = x.shape[0]
    d = x if torch.is_tensor(x) else torch.from_numpy(x).cuda()
    cell, order = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    off = torch.full((nel + 1,), -1, dtype=torch.int32, device="cuda")
    out, msg = C.c_int64(-1), C.c_char_p()
    rc = abi.load_library().gg_locate_noalloc(C.byref(mesh), n, d.data_ptr(), cell.data_ptr(), off.data_ptr(),
                                              order.data_ptr(), C.byref(out), None, C.byref(msg))
    return rc, cell, off, order, (msg.value or b"").decode()


def swarm(counts, seed):
    """counts[e] points in element e of a row of len(counts) elements, shuffled."""
    rng = np.random.default_rng(seed)
    e = rng.permutation(np.repeat(np.arange(len(counts)), counts))
    x = np.stack([(e + rng.uniform(0.01, 0.99, e.size)) / len(counts), rng.uniform(0.01, 0.99, e.size)], 1)
    return np.ascontiguousarray(x), e


@pytest.mark.parametrize("counts", [[1], [16] * 3 + [0, 15], [0, 17, 32, 1] * 40, [33, 64, 2] * 50, [65] + [3] * 200,
                                    [1024, 0, 700, 64], [40] * 300], ids=lambda c: f"{len(c)}x{max(c)}")
def test_sorted_order(counts):
    mesh = Mesh(2, (len(counts), 1))
    x, e = swarm(counts, max(counts))
    expect, offs = np.argsort(e, kind="stable"), np.concatenate([[0], np.cumsum(counts)])
    rc, cell, off, order, msg = noalloc(mesh, x, len(counts))
    assert rc == abi.GG_OK, msg
    assert np.array_equal(cell.cpu().numpy(), e)
    assert np.array_equal(off.cpu().numpy(), offs) and np.array_equal(order.cpu().numpy(), expect)
    # the handle's path: cells, and ξ of every point through the sorted arrays
    G = StokesProblem(mesh)
    G.set_points(x, (e % 3).astype(np.int32), x[:, 1].copy())
    assert np.array_equal(G.locate(), e)
    xi, w = G.integration_points()
    h = 1.0 / len(counts)
    assert np.allclose(xi[:, 0], 2 * (x[:, 0] - e * h) / h - 1, rtol=0, atol=1e-9)
    assert np.array_equal(w, 4.0 / np.asarray(counts)[e])


def test_more_points_than_an_element_may_hold():
    x, e = swarm([1025, 3], 1)
    rc, cell, off, order, msg = noalloc(Mesh(2, (2, 1)), x, 2)
    assert rc == abi.GG_ERR_INVALID and "1024" in msg
    assert np.array_equal(cell.cpu().numpy(), e) and off.cpu().tolist() == [0, 1025, 1028]
    x, e = swarm([5000, 3], 2)  # more than a place can count: still refused, the cells still right
    rc, cell, off, order, msg = noalloc(Mesh(2, (2, 1)), x, 2)
    assert rc == abi.GG_ERR_INVALID and np.array_equal(cell.cpu().numpy(), e)
    G = StokesProblem(Mesh(2, (2, 1)))  # a handle takes them
    G.set_points(x)
    assert np.array_equal(G.locate(), e)


def test_two_windows():
    torch = pytest.importorskip("torch")
    n, m = 17_000_001, 512
    x = torch.rand(n, 2, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    rc, cell, off, order, msg = noalloc(Mesh(2, (m, m)), x, m * m)
    assert rc == abi.GG_OK, msg
    e = (x * m).long().clamp_(max=m - 1)
    e = e[:, 0] + m * e[:, 1]
    assert torch.equal(cell.long(), e)
    assert torch.equal(order.long(), torch.sort(e, stable=True).indices)
    assert torch.equal(off[1:].long(), torch.bincount(e, minlength=m * m).cumsum(0))


def test_point_outside_is_refused():
    G = StokesProblem(Mesh(2, (2, 2)))
    G.set_points(np.array([[0.5, 0.25], [1.5, 0.5]]))
    with pytest.raises(GaleError):
        G.locate()


@pytest.mark.parametrize("nel,mean", [(3, 300), (700, 45), (70, 41), (5, 1300), (20000, 39), (30000, 3), (90000, 2)])
def test_blocks_of_few_and_many_elements(nel, mean):
    """The elements a block takes follow the mean count and the mesh: one per warp from 41
    points on, 32 to 128 below; single elements far from the mean in each, up to more than
    the in-place sort takes (the handle's path only)."""
    rng = np.random.default_rng(nel)
    counts = rng.poisson(mean, nel)
    counts[:: max(nel // 7, 1)] *= 3
    counts = np.maximum(counts, 1)
    x, e = swarm(counts, nel)
    mesh = Mesh(2, (nel, 1))
    expect, offs = np.argsort(e, kind="stable"), np.concatenate([[0], np.cumsum(counts)])
    rc, cell, off, order, msg = noalloc(mesh, x, nel)
    if counts.max() <= 1024:
        assert rc == abi.GG_OK, msg
        assert np.array_equal(off.cpu().numpy(), offs) and np.array_equal(order.cpu().numpy(), expect)
    else:
        assert rc != abi.GG_OK
    G = StokesProblem(mesh)
    G.set_points(x, (e % 3).astype(np.int32), x[:, 1].copy())
    assert np.array_equal(G.locate(), e)
    xi, w = G.integration_points()
    h = 1.0 / nel
    assert np.allclose(xi[:, 0], (x[:, 0] - (e + 0.5) * h) / (0.5 * h), atol=1e-9 * nel)
    assert np.array_equal(w, 4.0 / counts[e])


def test_dense_swarm_is_not_sorted_by_a_few_warps():
    """1000 points in each of 32² elements: 0.4 ms on a B200; blocks of 128 elements took 7.3."""
    mesh = Mesh(2, (32, 32))
    x = np.random.default_rng(5).random((1024 * 1000, 2))
    G = StokesProblem(mesh)
    G.set_points(x)
    best = 1.0
    for _ in range(200):  # a busy host delays single calls
        t = time.perf_counter()
        assert G.lib.gg_locate(G.h, None) == abi.GG_OK
        best = min(best, time.perf_counter() - t)
        if best < 2.5e-3:
            break
    assert best < 2.5e-3
