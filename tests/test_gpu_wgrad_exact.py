"""The training step's gradients on whole numbers: inputs, weights and output
gradients are small integers, so that every activation and propagated
gradient is exact in BF16 and every sum exact in FP32 in any order.  The
gradients then equal a 64-bit reference's to the last bit: a voxel left out or
counted twice at the edge of a tile shows, however large the crop."""
import numpy as np
import pytest

import wsnet_ref

pytestmark = pytest.mark.gpu


def integer_params(rng, nparam):
    """three weights of -1 or 1 per hidden channel, one per input channel of
    the output layer; no biases"""
    p, off = np.zeros(nparam, dtype=np.float32), 0
    for cin, cout in ((16, 24), (24, 24), (24, 24), (24, 1)):
        w = np.zeros((27, cout, cin), dtype=np.float32)
        if cout > 1:
            for co in range(cout):
                for q in rng.choice(27 * cin, 3, replace=False):
                    w[q % 27, co, q // 27] = rng.choice((-1.0, 1.0))
        else:
            w[rng.integers(0, 27, cin), 0, np.arange(cin)] = rng.choice((-1.0, 1.0), cin)
        p[off:off + w.size] = w.ravel()
        off += w.size + cout
    assert off == nparam
    return p


def exact(torch, params, x, k):
    """gradients for the output gradient k, in 64 bits"""
    layers = [W.reshape(3, 3, 3, W.shape[1], W.shape[2]).permute(3, 4, 0, 1, 2).double()
              for W, _ in wsnet_ref.split(params)]
    acts = [x.double().permute(0, 4, 1, 2, 3)]
    for L, w in enumerate(layers):
        z = torch.nn.functional.conv3d(acts[-1], w, padding=1)
        acts.append(torch.relu(z) if L < 3 else z)
    dz, grads = torch.from_numpy(k)[:, None].double(), []
    for L in (3, 2, 1, 0):
        assert acts[L].abs().max() <= 256 and dz.abs().max() <= 256  # exact in BF16
        gw = torch.nn.grad.conv3d_weight(acts[L], layers[L].shape, dz, padding=1)
        grads.append((gw.permute(2, 3, 4, 0, 1).reshape(-1), dz.sum((0, 2, 3, 4))))
        if L:
            dz = torch.nn.grad.conv3d_input(acts[L].shape, layers[L], dz, padding=1) * (acts[L] > 0)
    g = np.concatenate([v.numpy() for pair in reversed(grads) for v in pair])
    assert np.abs(g).max() < 2**24
    return acts[4][:, 0].numpy(), g


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 1, 3, 2), (1, 4, 16, 8), (3, 5, 17, 9), (1, 3, 15, 23),
                                   (2, 8, 32, 16), (8, 20, 40, 40), (5, 24, 48, 48), (3, 33, 49, 41)])
def test_gradients_of_whole_numbers_are_exact(ss4d, cuda, shape):
    torch = cuda
    nf, nz, ny, nx = shape
    rng = np.random.default_rng(nx)
    x = torch.from_numpy(rng.integers(-1, 2, (nf, nz, ny, nx, 16)).astype(np.float32)).to(torch.bfloat16)
    k = rng.integers(-1, 2, shape).astype(np.float32)
    with ss4d.Wsnet(seed=7) as net:
        params = integer_params(rng, net.nparam)
        net.set_params(params)
        y, want = exact(torch, params, x, k)
        # the step's output gradient 2 (y - t) / voxels rounds to k in BF16
        t = (y - k * (k.size / 2)).astype(np.float32)
        grad = torch.full((net.nparam,), float("nan"), dtype=torch.float32, device="cuda")
        net.train_step(ss4d.features_to_planar(x).cuda(), torch.from_numpy(t).cuda(), nx, ny, nz, nf, margin=0, lr=0.0,
                       grad=grad)
        net.check()
    assert np.array_equal(grad.cpu().numpy().astype(np.float64), want)
