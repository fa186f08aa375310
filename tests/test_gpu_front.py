"""The persistent presmoothing and the folded g faces at the edges of their
layouts: one to five columns (pairs of a colour, half-filled last pairs, both
row phases), one row, plane or frame, odd and even plane counts (the g
faces' fold in k), one and two images, spacings that are no power of two.
FP64: the oracle's bits; mixed: float-float arithmetic, whose operations
keep 2^-47 and whose sums and differences of values below 1 carry it into
K (grad)^2 with a factor below 4 K |grad| g^2 <= 130: 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1, 1), (2, 1, 1, 1), (3, 2, 1, 2), (4, 3, 2, 1), (5, 1, 3, 2), (33, 3, 5, 2), (34, 4, 4, 3), (67, 2, 7, 1)]


@pytest.mark.parametrize("h", [1.0, 0.125, 0.7, 3e-7])
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("images", [1, 2])
@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_edge_detector_matches_oracle(ss4d, oracle, cuda, dims, images, arith, h):
    torch = cuda
    rng = np.random.default_rng(sum(dims))
    shape = tuple(n + 2 for n in dims[::-1])
    img, thr = rng.random(shape), (rng.random(shape) > 0.7).astype(np.float64)
    # sigma follows h, so that the smoothing (sigma / h^2) is the usual one
    p = ss4d.scene_params(h=h, sigma=0.5 * h * h, K=1000.0 * h * h, gsTol=1e-9 * h ** 4, theta_img=0.5,
                          rho_thr=0.5 if images == 2 else 0.0)
    want_i, want_t = img.copy(), (thr.copy() if images == 2 else np.zeros(shape))
    want_g, (z0, z1), _ = oracle.edge_detector(p, want_i, want_t)
    i0 = torch.from_numpy(img).cuda()
    t0 = torch.from_numpy(thr).cuda() if images == 2 else None
    g = [torch.zeros_like(i0) for _ in range(8)]
    one = torch.from_numpy(img).cuda()
    prev = torch.empty_like(one)
    with ss4d.Solver(*shape[::-1], arith=arith) as S:
        S.edge_detector(p, i0, t0, g)
        st = S.presmooth_step(p, one, prev)
        faces = [torch.zeros_like(one) for _ in range(8)]
        S.gfaces(p, i0, t0, faces)
    assert st["iterations"] == z0
    assert np.array_equal(prev.cpu().numpy(), img)
    assert torch.equal(one, i0)
    inner = (slice(1, -1),) * 4
    got = [i0.cpu().numpy()] + ([t0.cpu().numpy()] if images == 2 else [])
    for a, b in zip(got, [want_i, want_t]):
        if arith == "fp64":
            assert np.array_equal(a, b)  # ghosts included
        else:
            assert np.abs(a - b).max() <= 1e-12
    for f in range(8):
        a, b, c = g[f].cpu().numpy()[inner], want_g[f][inner], faces[f].cpu().numpy()[inner]
        if arith == "fp64":
            assert np.array_equal(a, b) and np.array_equal(c, b), f
        else:
            assert np.abs(a - b).max() <= 1e-12 and np.abs(c - b).max() <= 1e-12, f
