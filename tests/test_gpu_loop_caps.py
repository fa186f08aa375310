"""The persistent loop on a capped grid: caps that leave just under and just
over two rounds per phase, where the targets are dealt out differently, in the
form whose last warp has no targets, and caps of the plain form (a volume of
more than three rounds).  Every target's arithmetic is the same, the sums'
order is not: the same u bit for bit, the same counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (37, 11, 13, 5): 13,585 columns and 7,150 pairs; 480 threads with targets per
# block: two rounds hold them from 15 and 8 blocks on.  (96, 64, 60, 10): 1.8e6
# and 0.9e6, on 304 blocks of 512 threads six to twelve rounds.
CASES = [((37, 11, 13, 5), [1, 2, 7, 8, 14, 15]), ((96, 64, 60, 10), [3, 150, 303])]


@pytest.mark.parametrize("dims,caps", CASES)
@pytest.mark.parametrize("arith", ["fp64", "mixed"])
def test_capped_grid_changes_nothing(ss4d, cuda, dims, caps, arith):
    torch = cuda
    p = ss4d.scene_params()
    _, u0 = ss4d.scene(1, *dims, seed=2)
    rng = np.random.default_rng(2)
    g = [torch.from_numpy(rng.uniform(0.05, 1.0, u0.shape)).cuda() for _ in range(8)]
    got = []
    for cap in [0] + caps:
        u = torch.from_numpy(u0).cuda()
        with ss4d.Solver.for_interior(*dims, arith=arith) as S:
            S.set_tiling(1, cap)
            st = S.seg_time_step(p, u, None, g)
        got.append((st["iterations"], st["refinements"], u))
    for it, ref, u in got[1:]:
        assert (it, ref) == got[0][:2]
        assert torch.equal(u, got[0][2])
