"""Failure detection in the persistent launches of a handle, without a fault:
with arrival counts that no arrival completes, the first wait of every block
runs out after about a second.  A step returns SS4D_ERR_TIMEOUT, u and the
context are as they were, and the next steps equal those of a handle whose
history of changes is empty.  Volumes of one round (the form whose last warp
has no targets) and of many; presmoothing and edge detector."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gives_up(ss4d, S, call):
    S.set_test_withhold_barrier(True)
    with pytest.raises(ss4d.SS4DError) as ei:
        call()
    assert ei.value.status == 5  # SS4D_ERR_TIMEOUT
    S.set_test_withhold_barrier(False)


@pytest.mark.parametrize("form", ["fp64", "mixed", "projected"])
@pytest.mark.parametrize("dims", [(20, 11, 9, 4), (96, 64, 60, 10)])
def test_step_gives_up_and_recovers(ss4d, cuda, form, dims):
    torch = cuda
    p = ss4d.scene_params()
    _, u0 = ss4d.scene(1, *dims, seed=2)
    rng = np.random.default_rng(2)
    g = [torch.from_numpy(rng.uniform(0.05, 1.0, u0.shape)).cuda() for _ in range(8)]

    def handle():
        S = ss4d.Solver.for_interior(*dims, arith="fp64" if form == "fp64" else "mixed")
        if form == "projected":
            S.set_extrapolation(3)
            S.set_projection(True)
        return S

    u = torch.from_numpy(u0).cuda()
    with handle() as S, handle() as F:
        for _ in range(4 if form == "projected" else 1):
            S.seg_time_step(p, u, None, g)
        before = u.clone()
        _gives_up(ss4d, S, lambda: S.seg_time_step(p, u, None, g))
        assert torch.equal(u, before)
        for _ in range(4 if form == "projected" else 1):
            a, b = S.seg_time_step(p, u, None, g), F.seg_time_step(p, before, None, g)
            assert (a["iterations"], a["projected"], a["residual"]) == (b["iterations"], b["projected"], b["residual"])
            assert torch.equal(u, before)


@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_batch_drops_the_history(ss4d, cuda, arith):
    """the batch's steps after a give-up start as a fresh batch's"""
    torch = cuda
    dims = [(20, 11, 9, 4), (13, 14, 8, 3)]
    p, us, gs = ss4d.scene_params(), [], []
    rng = np.random.default_rng(3)
    for d in dims:
        _, u0 = ss4d.scene(1, *d, seed=3)
        us.append(torch.from_numpy(u0).cuda())
        gs.append([torch.from_numpy(rng.uniform(0.05, 1.0, u0.shape)).cuda() for _ in range(8)])

    def batch():
        B = ss4d.Batch([tuple(n + 2 for n in d) for d in dims])
        if arith == "mixed":
            B.set_arith("mixed")
            B.set_extrapolation(3)
            B.set_projection(True)
        return B

    with batch() as B, batch() as F:
        for _ in range(3):
            B.seg_time_step([p, p], us, gs)
        before = [u.clone() for u in us]
        B.set_test_withhold_barrier(True)
        with pytest.raises(ss4d.SS4DError) as ei:
            B.seg_time_step([p, p], us, gs)
        assert ei.value.status == 5
        B.set_test_withhold_barrier(False)
        assert all(torch.equal(a, b) for a, b in zip(us, before))
        for _ in range(4):
            a, b = B.seg_time_step([p, p], us, gs), F.seg_time_step([p, p], before, gs)
            assert [s["iterations"] for s in a] == [s["iterations"] for s in b]
            assert all(torch.equal(x, y) for x, y in zip(us, before))


@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_edge_detector_gives_up_and_recovers(ss4d, cuda, arith):
    torch = cuda
    dims = (33, 9, 14, 7)
    i0, _ = ss4d.scene(1, *dims, seed=4)
    p = ss4d.scene_params()
    img = torch.from_numpy(i0).cuda()
    out = []
    with ss4d.Solver.for_interior(*dims, arith=arith) as S:
        for fail in (True, False):
            a, b = img.clone(), (img > 0.5).double()
            g = [torch.zeros_like(img) for _ in range(8)]
            if fail:
                _gives_up(ss4d, S, lambda: S.presmooth_step(p, img.clone()))
                _gives_up(ss4d, S, lambda: S.edge_detector(p, img.clone(), b.clone(), g))
            S.edge_detector(p, a, b, g)
            out.append([a, b] + [x[1:-1, 1:-1, 1:-1, 1:-1].clone() for x in g])
    assert all(torch.equal(x, y) for x, y in zip(*out))
