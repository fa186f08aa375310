"""The batch's per-volume kernels run on several streams between the caller's:
work pending on the caller's stream comes before them, what follows the call
after, and volumes that share memory keep the order of their numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _volumes(ss4d, torch, n, arith):
    out = []
    for v in range(n):
        dims = (20 + 3 * v, 18, 9 + v, 4) if v != 2 else (20, 18, 9, 4)
        p = ss4d.scene_params(K=600.0 + 100 * v)
        _, u0 = ss4d.scene(1, *dims, seed=3 + v)
        rng = np.random.default_rng(v)
        g = [torch.from_numpy(rng.uniform(0.05, 1.0, u0.shape)).cuda() for _ in range(8)]
        out.append((p, torch.from_numpy(u0).cuda(), g, dims))
    return out


def _single(ss4d, vol, arith, steps):
    p, u0, g, dims = vol
    u = u0.clone()
    with ss4d.Solver.for_interior(*dims, arith=arith) as S:
        for _ in range(steps):
            S.seg_time_step(p, u, None, g)
    return u


@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_work_pending_on_the_callers_stream(ss4d, cuda, arith):
    torch = cuda
    vols = _volumes(ss4d, torch, 6, arith)
    want = [_single(ss4d, v, arith, 2) for v in vols]
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with ss4d.Batch([tuple(n + 2 for n in v[3]) for v in vols], stream=st.cuda_stream) as B:
        B.set_arith(arith)
        with torch.cuda.stream(st):
            busy = torch.zeros(1 << 27, device="cuda")
            for _ in range(20):
                busy += 1.0  # about 3 ms ahead of the volumes' inputs
            us = [v[1].clone() for v in vols]
            for _ in range(2):
                B.seg_time_step([v[0] for v in vols], us, [v[2] for v in vols])
            got = [u.clone() for u in us]
        st.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_volumes_that_share_u(ss4d, cuda, arith):
    """both start from the shared u; the later one's result stays"""
    torch = cuda
    vols = _volumes(ss4d, torch, 5, arith)
    vols[2] = (vols[2][0], vols[0][1], vols[2][2], vols[2][3])
    want = [_single(ss4d, v, arith, 1) for v in vols]
    us = [v[1].clone() for v in vols]
    us[2] = us[0]
    with ss4d.Batch([tuple(n + 2 for n in v[3]) for v in vols]) as B:
        B.set_arith(arith)
        B.seg_time_step([v[0] for v in vols], us, [v[2] for v in vols])
    for v in (1, 2, 3, 4):
        assert torch.equal(us[v], want[v]), v
