"""The assemblies at the edges of their tiles, marches and folds: rows and
columns one short of, at and one past a tile, tiles of every width, one plane
or frame, odd and even plane counts (the mixed form's fold in k), a march of
several planes with a remainder, h a power of two, 1 and neither.  A step to
a tight tolerance against the oracle's: FP64 within the 1e-10 bar (the same
iterations), mixed (coefficients to about 1e-13, 35 voxel updates' worth of
them) within 1e-10 of the solution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(31, 7, 3, 2), (32, 8, 4, 1), (33, 9, 5, 3), (8, 33, 2, 2), (9, 31, 1, 3), (17, 16, 6, 2), (40, 5, 7, 2),
        (1, 40, 9, 1), (16, 9, 2, 2), (47, 7, 3, 2), (48, 8, 2, 3), (64, 64, 41, 4)]


@pytest.mark.parametrize("h", [1.0, 0.5, 0.8])
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_step_on_tile_edges_matches_oracle(ss4d, oracle, cuda, dims, arith, h):
    torch = cuda
    if dims[0] * dims[1] > 2000 and h != 1.0:
        pytest.skip("the long march once")
    rng = np.random.default_rng(dims[0])
    shape = tuple(n + 2 for n in dims[::-1])
    p = ss4d.scene_params(h=h, gsTol=1e-18 * h ** 4)
    u = rng.random(shape)
    g = [rng.uniform(0.05, 1.0, shape) for _ in range(8)]
    for d in range(4):  # a face between two interior voxels has one g, stored with both
        ax = 3 - d
        lo, hi = [slice(None)] * 4, [slice(None)] * 4
        lo[ax], hi[ax] = slice(1, -2), slice(2, -1)
        g[2 * d + 1][tuple(hi)] = g[2 * d][tuple(lo)]
    want = u.copy()
    z, _ = oracle.seg_time_step(p, want, np.zeros(shape), g, mmask=np.ones(shape))
    d = torch.from_numpy(u).cuda()
    with ss4d.Solver(*shape[::-1], arith=arith) as S:
        st = S.seg_time_step(p, d, None, [torch.from_numpy(a).cuda() for a in g])
    if arith == "fp64":
        assert st["iterations"] == z
    assert np.abs(d.cpu().numpy() - want).max() <= 1e-10 * np.abs(want).max()
