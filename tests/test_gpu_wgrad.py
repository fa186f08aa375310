"""The tensor-core weight gradient at the edges of its tiles (8 x 16 x 2
voxels): crops smaller than a tile, partial tiles along every axis, one frame
and several tiles per CTA (whose accumulators carry over).  The reference
rounds to BF16 where the kernels do (weights, activations, the propagated
gradients), so that only the order of FP32 sums and the roundings it flips
differ, also where a bias gradient's terms cancel: 2e-2 of each gradient's
norm."""
import numpy as np
import pytest

import wsnet_ref

pytestmark = pytest.mark.gpu


def reference(torch, params, x, t):
    layers = [(wsnet_ref.bf16(W.reshape(3, 3, 3, W.shape[1], W.shape[2]).permute(3, 4, 0, 1, 2)), b)
              for W, b in wsnet_ref.split(params)]
    acts = [x.float().permute(0, 4, 1, 2, 3)]
    for L, (w, b) in enumerate(layers):
        z = torch.nn.functional.conv3d(acts[-1], w, b, padding=1)
        acts.append(wsnet_ref.bf16(torch.relu(z)) if L < 3 else z)
    dz = wsnet_ref.bf16(2.0 * (acts[4] - torch.from_numpy(t)[:, None]) / t.size)
    grads = []
    for L in (3, 2, 1, 0):
        w = layers[L][0]
        gw = torch.nn.grad.conv3d_weight(acts[L], w.shape, dz, padding=1)
        grads.append((gw.permute(2, 3, 4, 0, 1).reshape(-1), dz.sum((0, 2, 3, 4))))
        if L:
            da = torch.nn.grad.conv3d_input(acts[L].shape, w, dz, padding=1)
            dz = wsnet_ref.bf16(da * (acts[L] > 0))
    return [v.numpy() for g in reversed(grads) for v in g]


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 1, 3, 2), (1, 4, 16, 8), (3, 5, 17, 9), (1, 3, 15, 23),
                                   (2, 8, 32, 16), (8, 20, 40, 40), (5, 24, 48, 48)])
def test_weight_gradient_matches_reference(ss4d, cuda, shape):
    torch = cuda
    nf, nz, ny, nx = shape
    rng = np.random.default_rng(nx)
    x = torch.from_numpy(rng.standard_normal((nf, nz, ny, nx, 16)).astype(np.float32)).to(torch.bfloat16)
    t = rng.standard_normal((nf, nz, ny, nx)).astype(np.float32)
    with ss4d.Wsnet(seed=7) as net:
        params = net.get_params()
        grad = torch.full((net.nparam,), float("nan"), dtype=torch.float32, device="cuda")
        net.train_step(ss4d.features_to_planar(x).cuda(), torch.from_numpy(t).cuda(), nx, ny, nz, nf, margin=0, lr=0.0,
                       grad=grad)
        g = grad.cpu().numpy().astype(np.float64)
        net.check()
    off = 0
    for want in reference(torch, params, x, t):
        assert np.linalg.norm(g[off:off + want.size] - want) <= 2e-2 * np.linalg.norm(want)
        off += want.size
