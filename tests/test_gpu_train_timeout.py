"""Failure detection in a training step, without a fault: with their loads
withheld, the weight gradients' waits (or all kernels') run out after about a
second each.  The step returns SS4D_ERR_TIMEOUT, its gradient is NaN, the
parameters stay as they were, and the steps after it equal those of a network
that never failed: neither the moments nor the step count moved."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("only", [True, False])
def test_train_step_timeout_is_reported_and_changes_nothing(ss4d, cuda, only):
    torch = cuda
    nf, nz, ny, nx = 2, 5, 17, 9
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.standard_normal((nf, nz, ny, nx, 16)).astype(np.float32)).to(torch.bfloat16)
    x = ss4d.features_to_planar(x).cuda()
    t = torch.from_numpy(rng.standard_normal((nf, nz, ny, nx)).astype(np.float32)).cuda()
    after = []
    for fail in (True, False):
        with ss4d.Wsnet(seed=7) as net:
            net.train_step(x, t, nx, ny, nz, nf, lr=1e-3)
            if fail:
                before = net.get_params()
                grad = torch.zeros(net.nparam, dtype=torch.float32, device="cuda")
                net.set_test_withhold_loads(True, weight_gradients_only=only)
                with pytest.raises(ss4d.SS4DError) as ei:
                    net.train_step(x, t, nx, ny, nz, nf, lr=1e-3, grad=grad)
                assert ei.value.status == 5  # SS4D_ERR_TIMEOUT
                with pytest.raises(ss4d.SS4DError):
                    net.check()
                net.set_test_withhold_loads(False)
                assert torch.isnan(grad).all()
                assert np.array_equal(net.get_params(), before)
            loss = [net.train_step(x, t, nx, ny, nz, nf, lr=1e-3) for _ in range(3)]
            net.check()
            after.append((loss, net.get_params()))
    assert after[0][0] == after[1][0]
    assert np.array_equal(after[0][1], after[1][1])
