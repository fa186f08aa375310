"""The rescale's cluster per frame: radii whose boundary passes through voxel
centres (the squared test must decide as the square root does), overlapping
balls, a box of one voxel, rows beyond the tables of the box (longer than 256
voxels), frames without balls, NaN inside a ball: the oracle's bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # interior, radius, balls (frame, x, y, z)
    ((20, 18, 16, 3), 5.0, [(1, 8.0, 9.0, 8.0), (1, 10.0, 9.0, 9.0), (3, 9.5, 8.25, 8.75)]),
    ((20, 18, 16, 2), 4.1231056256176606, [(1, 9.0, 9.0, 8.0), (2, 9.0, 9.0, 8.0), (2, 9.0, 9.0, 8.0)]),
    ((9, 9, 9, 1), 0.3, [(1, 4.0, 5.0, 4.0)]),
    ((40, 36, 34, 2), 14.5, [(2, 20.1, 18.3, 17.2), (2, 19.0, 17.0, 16.0)]),
    ((266, 264, 262, 1), 130.25, [(1, 133.0, 132.0, 131.5)]),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("nan", [False, True])
def test_rescale_matches_oracle(ss4d, oracle, cuda, case, nan):
    torch = cuda
    dims, R, balls = CASES[case]
    shape = tuple(n + 2 for n in dims[::-1])
    rng = np.random.default_rng(case)
    v = rng.standard_normal(shape) * 0.3 + 0.4
    mask = (rng.random(shape) > 0.1).astype(np.float64)
    if nan:
        l, x, y, z = balls[0]
        v[l, int(z), int(y), int(x)] = np.nan
    p = ss4d.scene_params(ballRadius=R)
    d = torch.from_numpy(v.copy()).cuda()
    with ss4d.Solver(*shape[::-1]) as S:
        S.rescale_to_zero_one(p, d, torch.from_numpy(mask).cuda(), balls)
    assert oracle.rescale(R, v, mask, balls) == 0
    assert np.array_equal(d.cpu().numpy(), v, equal_nan=True)
