"""The presmoothing's stop test at the tolerance: its residual differs from the
reference's in rounding (and in the order of the sum), so with gsTol set to
the very sum on which the reference stops it may go on, or stop one iteration
apart; such a test is reported as near the tolerance, however small the
residuals are beside the image's values.  One that is 1 % away is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1, 1), (3, 2, 1, 2), (5, 4, 3, 2), (17, 5, 6, 3), (33, 20, 9, 4)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("arith", ["fp64", "mixed"])
@pytest.mark.parametrize("scale,h", [(1.0, 1.0), (255.0, 0.25)])
def test_stop_at_the_references_sum_is_reported(ss4d, oracle, cuda, dims, arith, scale, h):
    torch = cuda
    shape = tuple(n + 2 for n in dims[::-1])
    rng = np.random.default_rng(sum(dims))
    img = rng.random(shape) * scale
    with ss4d.Solver(*shape[::-1], arith=arith) as S:
        for z in (1, 2, 4, 8, 12, 16, 24, 32):
            oracle.set_threads(1)  # a serial sum, twice the same (torch may have set its own number since)
            p = ss4d.scene_params(h=h, sigma=0.5 * h * h, gsTol=0.0)
            p.maxNoGSIteration_sigma = float(z)
            zr, R = oracle.presmooth(p, img.copy())
            if R == 0.0:
                break
            assert zr == z
            p.maxNoGSIteration_sigma = 200.0
            p.gsTol = R
            if oracle.presmooth(p, img.copy())[0] != z:
                continue  # at the rounding's own level an earlier sum was as small
            st = S.presmooth_step(p, torch.from_numpy(img).cuda())
            assert st["near_tolerance"] == 1, (z, R, st)
            # residuals above 1e-8 of the image, where the float-float terms'
            # 2^-44 d = 3e-13 stays below 1e-4 of them
            if R > 1e-16 * scale**2 * np.prod(dims) * h**4:
                p.gsTol = R * 1.01
                assert S.presmooth_step(p, torch.from_numpy(img).cuda())["near_tolerance"] == 0, (z, R)
