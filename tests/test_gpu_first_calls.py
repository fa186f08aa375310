"""First calls from several threads at once, in a process of their own: what
the launches look up once per process (occupancies, attributes, the tensor
map's encoder) is looked up by whichever thread comes first, and every
thread's results are those of a thread alone."""
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import sys, threading
sys.path.insert(0, sys.argv[1])
import numpy as np, torch, ss4d
dims = (20, 11, 9, 4)
p = ss4d.scene_params()
_, u0 = ss4d.scene(1, *dims, seed=2)
rng = np.random.default_rng(2)
g = [torch.from_numpy(rng.uniform(0.05, 1.0, u0.shape)).cuda() for _ in range(8)]
x = torch.from_numpy(rng.standard_normal((2, 5, 17, 9, 16)).astype(np.float32)).to(torch.bfloat16)
x = ss4d.features_to_planar(x).cuda()
t = torch.from_numpy(rng.standard_normal((2, 5, 17, 9)).astype(np.float32)).cuda()
torch.cuda.synchronize()
N, out, start = 6, {}, threading.Barrier(6)
def work(me):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        u = torch.from_numpy(u0).cuda()
        s.synchronize()
        with ss4d.Solver.for_interior(*dims, arith="mixed", stream=s.cuda_stream) as S, ss4d.Wsnet(seed=3, stream=s.cuda_stream) as net:
            S.set_extrapolation(3)
            S.set_projection(True)
            if me < N:
                start.wait()
            its = [S.seg_time_step(p, u, None, g)["iterations"] for _ in range(4)]
            loss = [net.train_step(x, t, 9, 17, 5, 2) for _ in range(2)]
            out[me] = (its, loss, u.cpu().numpy(), net.get_params())
threads = [threading.Thread(target=work, args=(m,)) for m in range(N)]
[h.start() for h in threads]
[h.join() for h in threads]
work(N)
for m in range(N):
    assert out[m][:2] == out[N][:2], (m, out[m][:2], out[N][:2])
    assert np.array_equal(out[m][2], out[N][2]) and np.array_equal(out[m][3], out[N][3]), m
print("equal")
"""


def test_first_calls_of_several_threads(ss4d, cuda):
    r = subprocess.run([sys.executable, "-c", PROGRAM, PKG], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ))
    assert r.returncode == 0 and r.stdout.strip() == "equal", r.stdout + r.stderr
