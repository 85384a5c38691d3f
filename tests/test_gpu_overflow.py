"""The inverse's normalisation of a sum that overflows: the transform of a spike c on one orbit is
scaled so that the unnormalised sum at the spike, c V, is past the largest number while its
partial sums (half of it before the last stage of the unfold) are not.  The spike comes back
infinite, as v / V of an infinite v is, and every other point finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


@pytest.mark.parametrize("sg,n,precision,batch", [(229, 48, 4, 1), (229, 48, 4, 64), (229, 24, 4, 2), (229, 96, 4, 30), (229, 40, 4, 2),
                                                  (229, 32, 4, 1), (229, 20, 8, 1), (229, 40, 8, 2)])
def test_spike(cf, O, prep, sg, n, precision, batch):
    p, N = prep(sg, (n, n, n)), (n, n, n)
    plan = cf.KRFFTPlan(p["spec"], p["ops_s"], precision=precision, max_batch=batch)
    u = np.zeros(N)
    x = np.array([2, 4, 6])
    for op in p["oops"]:
        u[tuple(np.mod(np.asarray(op.Rm) @ x + np.asarray(op.tv), N))] = 1.0
    f0 = O.pack_stride(u, plan.L).T
    dt = torch.float32 if precision == 4 else torch.float64
    t = torch.tensor(np.ascontiguousarray(np.broadcast_to(f0, (batch,) + f0.shape)), dtype=dt, device="cuda")
    c = 1.4 * (torch.finfo(dt).max / np.prod(plan.M))
    back = plan.backward(plan.forward(t) * c).view(t.shape)
    spike = t > 0
    assert torch.isinf(back[spike]).all() and torch.isfinite(back[~spike]).all()
    plan.close()
