"""The persistent loop (one cooperative launch, every block running the
controller) against the host-driven loop of separate kernels: the same
arithmetic per target, so the same u bit for bit and the same counts, at the
edges of its flat walk (one voxel, odd rows, one row, a volume of one round
and of just over two rounds of the grid, whose last round is dealt out
differently) and through every phase (rounds from zero and from a projected
start, several rounds, given coefficients, the host-array step's pauses)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# two rounds of 304 blocks of 512 threads are 311,296 pairs (mixed) or
# columns (FP64): the first of each couple fills them, the second goes on
SIZES = [(1, 1, 1, 1), (2, 1, 3, 2), (3, 5, 1, 7), (33, 9, 14, 7), (47, 31, 23, 5), (64, 4, 4, 2),
         (64, 32, 38, 16), (65, 32, 38, 16), (64, 32, 38, 8), (65, 32, 38, 8),
         # one round and three rounds of the form whose last warp has no
         # targets (304 blocks of 480 columns, 152 of 480 pairs), and just over
         (64, 38, 12, 10), (65, 38, 12, 10), (64, 38, 36, 10), (65, 38, 36, 10)]


def _volume(ss4d, torch, dims, seed, **over):
    p = ss4d.scene_params(**over)
    i0, u0 = ss4d.scene(1, *dims, seed=seed)
    rng = np.random.default_rng(seed)
    g = [torch.from_numpy(rng.uniform(0.05, 1.0, i0.shape)).cuda() for _ in range(8)]
    return p, torch.from_numpy(u0).cuda(), g


@pytest.mark.parametrize("dims", SIZES)
@pytest.mark.parametrize("form", ["fp64", "mixed", "projected", "tight"])
def test_persistent_loop_equals_host_driven_loop(ss4d, cuda, dims, form):
    torch = cuda
    # tight: several rounds of corrections and refinement passes per step
    p, u0, g = _volume(ss4d, torch, dims, 3, **({"gsTol": 1e-20} if form == "tight" else {}))
    out = []
    for device_loop in (True, False):
        u = u0.clone()
        with ss4d.Solver.for_interior(*dims, arith="fp64" if form == "fp64" else "mixed") as S:
            S.set_graph(device_loop)
            if form == "projected":
                S.set_extrapolation(3)
                S.set_projection(True)
            rec = []
            for _ in range(4 if form == "projected" else 2):
                st = S.seg_time_step(p, u, None, g)
                rec.append((st["iterations"], st["refinements"], st["projected"]))
        out.append((rec, u.cpu().numpy()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("arith", ["fp64", "mixed"])
@pytest.mark.parametrize("dims", [(1, 1, 1, 1), (21, 6, 9, 4), (40, 20, 20, 20)])
def test_persistent_loop_on_given_coefficients(ss4d, cuda, dims, arith):
    """ss4d_sor_solve and the MCF step: the first refinement pass runs in the
    loop (no pass formed by the assembly)"""
    torch = cuda
    p, u0, _ = _volume(ss4d, torch, dims, 7)
    rng = np.random.default_rng(5)
    coef = [torch.from_numpy(rng.uniform(0.0, 1.0, tuple(u0.shape))).cuda() for _ in range(8)]
    prev = u0 + 0.01 * torch.from_numpy(rng.standard_normal(tuple(u0.shape))).cuda()
    m = ss4d.mcf_params(16, tau=0.01, eps2=1e-2, h=0.15)
    out = []
    for device_loop in (True, False):
        u, w = u0.clone(), u0.clone()
        with ss4d.Solver.for_interior(*dims, arith=arith) as S:
            S.set_graph(device_loop)
            its = [S.sor_solve(p, u, prev, coef)["iterations"], S.mcf_time_step(m, 1, w)["iterations"]]
        out.append((its, u.cpu().numpy(), w.cpu().numpy()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("max_grid", [1, 3, 0])
def test_persistent_loop_grid_cap(ss4d, cuda, max_grid):
    """a capped grid (down to one block, whose barriers are its own) changes nothing"""
    torch = cuda
    dims = (37, 11, 13, 5)
    p, u0, g = _volume(ss4d, torch, dims, 2)
    for arith in ("fp64", "mixed"):
        got = []
        for cap in (max_grid, 0):
            u = u0.clone()
            with ss4d.Solver.for_interior(*dims, arith=arith) as S:
                S.set_tiling(1, cap)
                st = S.seg_time_step(p, u, None, g)
            got.append((st["iterations"], u.cpu().numpy()))
        assert got[0][0] == got[1][0]
        assert np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("form,maxit", [("mixed", 200), ("mixed", 6), ("mixed", 9), ("projected", 200), ("tight", 200)])
def test_graph_loop_equals_host_driven_loop(ss4d, cuda, form, maxit):
    """Volumes above 5e6 voxels run the mixed loop as a graph whose bodies hold
    four iterations and whose half-sweep runs the controller: rounds that end
    at any of the four, a limit that ends the loop inside a body."""
    torch = cuda
    dims = (131, 127, 62, 5)
    p, u0, g = _volume(ss4d, torch, dims, 11, maxNoGSIteration=maxit, **({"gsTol": 1e-20} if form == "tight" else {}))
    out = []
    for device_loop in (True, False):
        u = u0.clone()
        with ss4d.Solver.for_interior(*dims, arith="mixed") as S:
            S.set_graph(device_loop)
            if form == "projected":
                S.set_extrapolation(3)
                S.set_projection(True)
            rec = []
            for _ in range(4 if form == "projected" else 2):
                st = S.seg_time_step(p, u, None, g)
                rec.append((st["iterations"], st["refinements"], st["projected"]))
        out.append((rec, u))
    assert out[0][0] == out[1][0]
    assert torch.equal(out[0][1], out[1][1])
