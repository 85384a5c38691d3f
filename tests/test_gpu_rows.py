"""The compile-time sized kernels at the edges of their dispatch: small launches (split
lines, rows of two slots), full rows of representatives with a remainder, every channel
edge, all centrings, and groups with screw axes, glides and no inversion centre, where the
fibers of the inverse gather carry phases and conjugated taps.  Each field is a seeded
combination of two symmetric oracle fields, so its spectrum is the same combination of two
FP64 full-grid FFTs (test/runtests.jl:199-216, test/test_centered_backward.jl:31-70).

Tolerances: the worst-case growth of a radix-r FFT pass is a few roundings, so a transform of
n points is within about 4 log2(n) eps of the largest value; 4 x 17 x 1.2e-7 = 8e-6 for FP32
at 48^3 points and 1.5e-14 for FP64, and the round trip doubles that.  The bars are 1e-5 and
2e-13, and twice that for the round trip."""
import numpy as np
import pytest

from conftest import q_plan, rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

TOL = {4: 1e-5, 8: 2e-13}


def check(cf, O, prep, sg, N, precision, batch):
    ps = [prep(sg, N, seed=s) for s in (31, 32)]
    plan = cf.KRFFTPlan(ps[0]["spec"], ps[0]["ops_s"], precision=precision, max_batch=batch)
    ospec = O.calc_spectral_asu(ps[0]["oops"], len(N), N)
    bases = np.stack([O.pack_stride(p["u"], plan.L) for p in ps])
    truths = np.stack([O.spectrum_on_asu(p["u"], ospec) for p in ps])
    coef = np.random.default_rng(batch).standard_normal((batch, 2))
    f0 = np.tensordot(coef, bases, 1)
    order = (0,) + tuple(range(len(N), 0, -1))
    x = torch.tensor(np.ascontiguousarray(f0.transpose(order)), device="cuda",
                     dtype=torch.float32 if precision == 4 else torch.float64)
    F = plan.forward(x)
    back = plan.backward(F).cpu().numpy().reshape(x.shape)
    F = F.cpu().numpy().reshape(batch, -1)
    for b in range(batch):
        assert rel_err(F[b], coef[b] @ truths) < TOL[precision], b
        assert rel_err(back[b], f0[b].T) < 2 * TOL[precision], b
    plan.close()


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("sg,n,batch", [(229, 16, 1), (229, 24, 3), (229, 32, 33), (230, 48, 2), (229, 48, 17), (227, 64, 9),
                                        (230, 64, 36), (225, 96, 5), (229, 96, 1), (47, 32, 70), (221, 48, 19)])
def test_channel_edges(cf, O, prep, sg, n, batch, precision):
    check(cf, O, prep, sg, (n, n, n), precision, batch)


@pytest.mark.parametrize("sg", [2, 16, 19, 23, 24, 62, 92, 96, 122, 141, 198, 199, 205, 212, 214, 220, 228])
def test_fiber_phases(cf, O, prep, sg):
    check(cf, O, prep, sg, (16, 16, 16), 8, 11)


def test_largest_edge(cf, O, prep):
    check(cf, O, prep, 221, (96, 96, 96), 4, 3)  # plain lattice, 48 points per line


@pytest.mark.parametrize("sg,n,batch,precision", [(47, 8, 1, 8), (47, 12, 3, 8), (200, 16, 2, 4), (221, 24, 40, 8), (47, 48, 2, 4),
                                                  (123, 64, 7, 8), (47, 96, 3, 4)])
def test_separable_step(cf, O, prep, sg, n, batch, precision):
    # both z transforms and the Q-multiply in one kernel: blocks of few and of all line pairs
    N, lat = (n, n, n), np.diag([1.0, 1.0, 1.3]) if sg == 123 else np.diag([1.0, 1.3, 0.8]) if sg == 47 else np.eye(3)
    p = prep(sg, N, seed=33)
    plan = q_plan(cf, p, cf.PATH_M2Q, 0.01, lat, precision=precision, max_batch=batch)
    assert plan.info.exec_path & 64
    f0 = O.pack_stride(p["u"], plan.L).T
    want = O.fullgrid_reference(p["u"], N, 0.01, lat, plan.L).T
    scale = np.arange(1, batch + 1).reshape(-1, 1, 1, 1)
    q = torch.tensor(scale * f0, device="cuda", dtype=torch.float32 if precision == 4 else torch.float64)
    plan.scft_step(q)
    for b in range(batch):
        assert rel_err(q[b].cpu().numpy(), (b + 1) * want) < 2 * TOL[precision], b
    plan.close()


@pytest.mark.parametrize("sg,N,batch,precision", [(47, (20, 24, 30), 3, 8), (47, (36, 50, 54), 2, 4), (47, (64, 32, 96), 1, 4),
                                                  (191, (9, 9, 25), 5, 8), (191, (27, 27, 10), 2, 8), (191, (45, 45, 16), 2, 4),
                                                  (229, (20, 20, 20), 9, 8), (229, (40, 40, 40), 4, 4), (225, (36, 36, 36), 17, 8),
                                                  (230, (72, 72, 72), 1, 4), (227, (80, 80, 80), 3, 4), (166, (12, 12, 30), 2, 8),
                                                  (123, (24, 24, 40), 2, 8), (221, (90, 90, 90), 1, 4), (62, (48, 20, 60), 33, 4)])
def test_general_shapes(cf, O, prep, sg, N, batch, precision):
    # radices 2 to 16 on every axis, one-factor and two-factor lengths, unequal axes, folds
    check(cf, O, prep, sg, N, precision, batch)


@pytest.mark.parametrize("sg,N,batch,precision", [(11, (30, 30), 1, 8), (11, (160, 160), 5, 8), (2, (18, 50), 3, 4), (17, (45, 45), 2, 8),
                                                  (9, (64, 24), 7, 4)])
def test_general_planes(cf, O, prep, sg, N, batch, precision):
    check(cf, O, prep, sg, N, precision, batch)


@pytest.mark.parametrize("sg,N,precision", [(229, (20, 20, 20), 8), (225, (30, 30, 30), 4), (47, (18, 10, 24), 8), (191, (9, 9, 5), 4)])
def test_grid_conversion_shapes(cf, O, prep, sg, N, precision):
    # whole grid -> subgrid -> whole grid of symmetric fields: copies, so equal to the bit
    p, batch = prep(sg, N, seed=34), 6
    plan = cf.KRFFTPlan(p["spec"], p["ops_s"], precision=precision, max_batch=batch)
    u = torch.tensor(np.ascontiguousarray(np.stack([(b + 1) * p["u"].T for b in range(batch)])), device="cuda",
                     dtype=torch.float32 if precision == 4 else torch.float64)
    L = plan.L
    f0 = plan.fullgrid_to_subgrid(u)
    assert torch.equal(f0, u[:, ::L[2], ::L[1], ::L[0]])
    back = plan.subgrid_to_fullgrid(f0)
    assert torch.max(torch.abs(back - u)).item() <= 1e-5 * torch.max(torch.abs(u)).item()
    assert torch.equal(back[:, ::L[2], ::L[1], ::L[0]], f0)
    shifted = torch.empty(u.numel() + 1, dtype=u.dtype, device="cuda")[1:].view(u.shape)  # unaligned output
    assert torch.equal(plan.subgrid_to_fullgrid(f0, out=shifted), back)
    plan.close()
