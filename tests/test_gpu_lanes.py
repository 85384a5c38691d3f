"""Dispatch by launch size: one or two concurrent lanes, split lines or a line per thread, rows of
two slots or full rows.  A batch on either side of each line gives the fields' own single-call
results, forward, backward and through two contour steps.

Tolerance: either result is within about 4 log2(n) eps of the largest value of a transform of n
points (4 x 18 x 1.1e-16 = 8e-15 at 64^3 points, 8.6e-6 in FP32), a contour step takes two
transforms: 2 x 2 x 2 x 8e-15 = 6e-14 and 7e-5.  The bars are 1e-13 and 1e-4."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from conftest import rel_err


@pytest.mark.parametrize("sg,N,precision,batches", [(229, (128, 128, 128), 8, (8, 17, 23, 25)), (225, (128, 128, 128), 8, (33, 37, 49)),
                                                    (221, (64, 64, 64), 8, (17, 65, 97)), (221, (64, 64, 64), 4, (16, 32)),
                                                    (1, (32, 32, 32), 8, (16, 64)), (1, (32, 32, 32), 4, (17,)),
                                                    (229, (96, 96, 96), 4, (12, 112)), (191, (60, 60, 80), 8, (3, 5)),
                                                    (229, (80, 80, 80), 4, (9, 33))])
def test_batches_equal_single_calls(cf, sg, N, precision, batches):
    dt, ct = (torch.float32, torch.complex64) if precision == 4 else (torch.float64, torch.complex128)
    bar = 1e-4 if precision == 4 else 1e-13
    _, ops = cf.find_optimal_shift(cf.get_ops(sg, 3, N), N)
    spec = cf.calc_spectral_asu(ops, 3, N)
    one = cf.KRFFTPlan(spec, ops, N=N, ds=0.01, precision=precision)
    g = torch.Generator(device="cuda").manual_seed(sg)
    for B in batches:
        plan = cf.KRFFTPlan(spec, ops, N=N, ds=0.01, precision=precision, max_batch=B)
        f0 = torch.randn((B,) + tuple(reversed(plan.M)), generator=g, device="cuda", dtype=dt)
        w = torch.rand(f0.shape, generator=g, device="cuda", dtype=dt)
        F = plan.forward(f0)
        back = plan.backward(F)
        q = plan.step_diffusion(f0.clone(), w, 0.01, 2)
        for b in {0, 1, B // 2, B - 2, B - 1}:
            x = f0[b].contiguous()
            G = one.forward(x)
            assert rel_err(F[b].cpu().numpy(), G.cpu().numpy()) < bar, (B, b)
            assert rel_err(back[b].cpu().numpy(), one.backward(G).cpu().numpy()) < bar, (B, b)
            assert rel_err(q[b].cpu().numpy(), one.step_diffusion(x, w[b].contiguous(), 0.01, 2).cpu().numpy()) < bar, (B, b)
        plan.close()
    one.close()
