"""The iteration limit at the ends of its range: "no limit" (2^30, 10^9 and the
largest int, where four bodies per iteration no longer fit 32 bits) ends where
a limit of 1000 does, and a limit of 0 or below where the reference's do-while
does: after one iteration in the FP64 form, at the first residual test in the
mixed form.  The persistent loop, the host-driven one, the host-array step and
the batch (persistent, graph, host-driven)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITS = [2**30, 10**9, 2**31 - 1, 0, -9, -10, -(2**31)]
DIMS = (21, 14, 9, 4)


def _scene(ss4d, seed=3):
    p = ss4d.scene_params()
    _, u0 = ss4d.scene(1, *DIMS, seed=seed)
    rng = np.random.default_rng(seed)
    return p, u0, [rng.uniform(0.05, 1.0, u0.shape) for _ in range(8)]


def _limit_alike(arith, limit):
    """a limit inside every type's range with the same meaning"""
    return 1000 if limit > 0 else (1 if arith == "fp64" else 0)


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("arith", ["fp64", "mixed"])
@pytest.mark.parametrize("route", ["device", "host", "arrays"])
def test_step(ss4d, cuda, arith, limit, route):
    from test_gpu_parity import _pinned

    torch = cuda
    p, u0, g = _scene(ss4d)
    dg = [torch.from_numpy(a).cuda() for a in g]
    out = []
    for maxit in (limit, _limit_alike(arith, limit)):
        p.maxNoGSIteration = maxit
        with ss4d.Solver.for_interior(*DIMS, arith=arith) as S:
            S.set_graph(route != "host")
            if route == "arrays":
                hu, free = _pinned(ss4d, u0.shape)
                hu[...] = u0
                st = S.seg_time_step_host(p, hu, torch.zeros_like(dg[0]), dg)
                u = hu.copy()
                free()
            else:
                d = torch.from_numpy(u0).cuda()
                st = S.seg_time_step(p, d, None, dg)
                u = d.cpu().numpy()
        out.append((st["iterations"], st["refinements"], st["residual"], u))
    assert out[0][:3] == out[1][:3]
    assert np.array_equal(out[0][3], out[1][3])
    if limit > 0:
        assert out[0][0] > 1 and out[0][2] <= p.gsTol
    else:
        assert out[0][0] == _limit_alike(arith, limit)


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("arith", ["fp64", "mixed"])
@pytest.mark.parametrize("loop", ["persistent", "graph", "host"])
def test_batch(ss4d, cuda, arith, limit, loop):
    torch = cuda
    p, u0, g = _scene(ss4d)
    dg = [torch.from_numpy(a).cuda() for a in g]
    out = []
    for maxit in (limit, _limit_alike(arith, limit)):
        p.maxNoGSIteration = maxit
        with ss4d.Batch([tuple(n + 2 for n in DIMS)] * 2) as B:
            if arith == "mixed":
                B.set_arith("mixed")
            B.set_persistent(loop == "persistent")
            B.set_graph(loop == "graph")
            us = [torch.from_numpy(u0).cuda() for _ in range(2)]
            st = B.seg_time_step([p, p], us, [dg, dg])
        out.append(([s["iterations"] for s in st], [s["residual"] for s in st], [u.cpu().numpy() for u in us]))
    assert out[0][:2] == out[1][:2]
    assert all(np.array_equal(a, b) for a, b in zip(out[0][2], out[1][2]))
    if limit > 0:
        assert all(r <= p.gsTol for r in out[0][1])
