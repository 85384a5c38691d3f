"""General kernels (channel grids without a compile-time sized kernel): the fields of a batch
do not see one another.  A field's result in a batch equals, to the bit, that of a call of its
own, whatever its neighbours hold: values 1e5 times larger, NaN, or spectra whose inverse is
not real (cfft_backward returns the real part; src/centering_fold.jl:745-775)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

SHAPES = [(229, (20, 20, 20), 4), (225, (36, 36, 36), 8), (191, (9, 9, 25), 8), (47, (36, 50, 54), 4), (1, (12, 20, 18), 8),
          (11, (30, 30), 4), (9, (64, 24), 8)]


@pytest.mark.parametrize("sg,N,precision", SHAPES)
def test_fields_independent(cf, prep, sg, N, precision):
    p, B = prep(sg, N), 5
    plan = cf.KRFFTPlan(p["spec"], p["ops_s"], precision=precision, max_batch=B)
    assert not plan.info.exec_path & 1
    rng = np.random.default_rng(sg)
    dt = torch.float32 if precision == 4 else torch.float64
    scale = np.array([1.0, 1e5, 1e-5, 1.0, 1.0])
    shape = (B,) + tuple(reversed(plan.M))
    f0 = torch.tensor(rng.standard_normal(shape) * scale.reshape((B,) + (1,) * len(N)), dtype=dt, device="cuda")
    F = torch.tensor((rng.standard_normal((B, plan.n_spec, 2)) * scale.reshape(B, 1, 1)), dtype=dt, device="cuda")
    f0.view(B, -1)[3, 0] = float("nan")
    F[3, 0, 0] = float("nan")
    F = torch.view_as_complex(F)
    G, g0 = plan.forward(f0), plan.backward(F)
    for b in (0, 1, 2, 4):
        assert torch.isfinite(torch.view_as_real(G[b])).all() and torch.isfinite(g0[b]).all(), b
        assert torch.equal(G[b], plan.forward(f0[b].contiguous())), b
        assert torch.equal(g0[b], plan.backward(F[b].contiguous())), b
    plan.close()
