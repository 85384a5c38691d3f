"""cfft_backward of any spectrum, not only of a real symmetric field's: G0 at every orbit
representative is the alias row of the plan's backward tables term by term (one value or its
conjugate per alias, src/krfft.jl:1285-1311, src/centering_fold.jl:782-813), each image of it
takes its phase from the first operation that reaches it, and f0 is the real part of the
inverse FFT.

Tolerance: values of a few, sums of 8 terms and an inverse transform of n points are within
about 4 log2(n) eps of the largest value: 4 x 13 x 1.2e-7 = 6e-6 for FP32 at 16^3 to 24 x 36
points, 1.2e-14 for FP64.  The bars are 1e-5 and 2e-13."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


def alias_rows(plan, oops, F):
    D, N, L, M = len(plan.N), plan.N, plan.L, plan.M
    reps, s_tab, p_tab = (np.asarray(v) for v in plan.backward_tables())
    P, d = int(np.lcm.reduce(N)), int(np.prod(L))
    v = np.where(s_tab != 0, F[np.maximum(np.abs(s_tab) - 1, 0)], 0.0)
    v = np.where(s_tab < 0, v.conj(), v) * np.exp(2j * np.pi * p_tab / P)
    vals = v.reshape(len(reps), d).sum(axis=1) / d
    q = np.stack(np.unravel_index(reps, M, order="F"))
    G0, done = np.zeros(int(np.prod(M)), dtype=complex), np.zeros(int(np.prod(M)), dtype=bool)
    for op in oops:
        R, t = np.asarray(op.Rm), np.asarray(op.tv)
        Rs = R * np.asarray(L)[None, :]
        if np.any(t % L) or np.any(Rs % np.asarray(L)[:, None]):
            continue
        R, s = Rs // np.asarray(L)[:, None], t // L
        at = np.ravel_multi_index(np.mod(R.T @ q, np.asarray(M)[:, None]), M, order="F")
        ph = np.exp(2j * np.pi * np.sum(q * s[:, None] / np.asarray(M)[:, None], axis=0))
        new = ~done[at]
        G0[at[new]] = (vals * ph)[new]
        done[at] = True
    return np.fft.ifftn(G0.reshape(M, order="F")).real


@pytest.mark.parametrize("sg,N,precision", [(229, (16, 16, 16), 8), (229, (16, 16, 16), 4), (229, (20, 20, 20), 8), (230, (24, 24, 24), 8),
                                            (227, (16, 16, 16), 8), (47, (16, 16, 16), 8), (47, (12, 18, 20), 4), (2, (16, 16, 16), 8),
                                            (62, (20, 20, 20), 8), (70, (20, 20, 20), 8), (186, (12, 12, 20), 8), (198, (16, 16, 16), 8),
                                            (11, (20, 20), 8), (9, (24, 36), 4)])
def test_backward_of_any_spectrum(cf, prep, sg, N, precision):
    p = prep(sg, N)
    plan = cf.KRFFTPlan(p["spec"], p["ops_s"], precision=precision)
    rng = np.random.default_rng(sg)
    F = rng.standard_normal(plan.n_spec) + 1j * rng.standard_normal(plan.n_spec)
    x = torch.tensor(F, dtype=torch.complex64 if precision == 4 else torch.complex128, device="cuda")
    got = plan.backward(x).cpu().numpy().astype(np.float64).T
    assert rel_err(got, alias_rows(plan, p["oops"], F)) < (1e-5 if precision == 4 else 2e-13)
    plan.close()
