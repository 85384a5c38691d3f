"""Contour steps on grids without a compile-time kernel: the interaction factors of the general
and of the Stockham kernels (src/diffusion_solver.jl:254-282), every field with a w of its own.
The truth is the full-grid recursion in FP64.

Tolerance: a step is two transforms of n points and two factors, each within about 4 log2(n) eps of
the largest value (4 x 17 x 1.2e-7 = 8e-6 in FP32, 1.5e-14 in FP64), and errors of random sign add
like the root of the number of steps: 2 x 5 x 8e-6 = 8e-5 after 24 steps, 1.5e-13.  The bars are 1e-4
and 5e-13, and 2e-5 and 1e-13 for the transforms."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DS, DT = 0.01, 0.02


def check(cf, O, prep, sg, N, precision, batch, steps, lat=None):
    D = len(N)
    lat = np.eye(D) * 3.0 if lat is None else lat
    fs = [prep(sg, N, seed=51 + s) for s in range(2)]
    p = fs[0]
    plan = cf.KRFFTPlan(p["spec"], p["ops_s"], N=N, ds=DS, lattice=lat, precision=precision, max_batch=batch)
    assert not plan.info.exec_path & 1
    rng = np.random.default_rng(sg)
    co = rng.uniform(0.5, 2.0, (batch, 2)) * np.where(np.arange(batch) % 2, 10.0, 1.0)[:, None]
    u = [a * fs[0]["u"] for a in co[:, 0]]
    w = [b * np.abs(fs[1]["u"]) for b in co[:, 1]]
    dt = torch.float32 if precision == 4 else torch.float64
    dev = lambda fields: torch.tensor(np.ascontiguousarray(np.stack([O.pack_stride(f, plan.L).T for f in fields])), dtype=dt, device="cuda")
    f0, wd = dev(u), dev(w)
    ospec = O.calc_spectral_asu(p["oops"], D, N)
    F = plan.forward(f0).cpu().numpy().reshape(batch, -1)
    back = plan.backward(plan.forward(f0)).view(f0.shape).cpu().numpy()
    one, many = plan.scft_step(f0.clone()).cpu().numpy(), plan.step_diffusion(f0.clone(), wd, DT, steps).cpu().numpy()
    tol, tol_t = (1e-4, 2e-5) if precision == 4 else (5e-13, 1e-13)
    kx = np.meshgrid(*[np.where(np.arange(n) >= n // 2, np.arange(n) - n, np.arange(n)) for n in N], indexing="ij")
    g = 2 * np.pi * np.linalg.inv(lat).T
    K = np.exp(-DS * sum(sum(g[i, j] * kx[j] for j in range(D)) ** 2 for i in range(D)))
    D_ = lambda x: np.fft.ifftn(K * np.fft.fftn(x)).real
    for b in range(batch):
        assert rel_err(F[b], O.spectrum_on_asu(u[b], ospec)) < tol_t, b
        assert rel_err(back[b], f0[b].cpu().numpy()) < 2 * tol_t, b
        assert rel_err(one[b], O.pack_stride(D_(u[b]), plan.L).T) < 2 * tol_t, b
        e, q = np.exp(-0.5 * DT * w[b]), u[b]
        for _ in range(steps):
            q = e * D_(e * q)
        assert rel_err(many[b], O.pack_stride(q, plan.L).T) < tol, b
    plan.close()


@pytest.mark.parametrize("sg,N,precision,batch,steps", [(229, (40, 40, 40), 4, 3, 24), (229, (20, 20, 20), 8, 5, 24), (225, (36, 36, 36), 8, 2, 7),
                                                        (47, (20, 24, 32), 4, 3, 24), (47, (12, 18, 20), 8, 2, 24), (221, (30, 30, 30), 8, 1, 3),
                                                        (11, (30, 30), 8, 3, 24), (2, (18, 50), 4, 2, 24)])
def test_general_steps(cf, O, prep, sg, N, precision, batch, steps):
    check(cf, O, prep, sg, N, precision, batch, steps)


# Channel lengths that do not split into two register radices (125 and 162), and phase
# denominators past the packed tables' 2048 (lcm(20, 54, 32) = 4320).
@pytest.mark.parametrize("sg,N,precision,batch,steps", [(47, (250, 6, 10), 8, 3, 7), (47, (8, 324, 6), 4, 2, 7), (47, (20, 54, 32), 8, 3, 7),
                                                        (16, (20, 54, 32), 4, 2, 24), (2, (20, 54, 32), 8, 2, 3), (2, (12, 162), 8, 3, 7)])
def test_stockham_steps(cf, O, prep, sg, N, precision, batch, steps):
    check(cf, O, prep, sg, N, precision, batch, steps)
