"""Dead points whose residual sum leaves the fp32 range: their weight is zero, the evidence is that of
the other points; the gradient, zero times an infinite residual, is not a number."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dead_set(M, P, N, over):
    from jaxns_gb300.adjoint import DeadSet
    g = np.random.default_rng(M + P)
    U = np.full((M, P), 0.5)
    U[over] = 1.0 - 1e-12  # w = 7 tau in every dimension
    dev = lambda x: torch.as_tensor(x, device="cuda")
    return DeadSet(U=dev(U), log_w=dev(g.standard_normal(M)), Phi=dev(np.ones((N, P), np.float32)),
                   y=dev(g.standard_normal(N).astype(np.float32)))


@pytest.mark.parametrize("P", [3, 40])
@pytest.mark.parametrize("tensor_cores", [True, False])
def test_overflowing_points_have_no_weight(gpu_lib, P, tensor_cores):
    """One overflowing point in every range of 128 (a range is a block of the reduction)."""
    from jaxns_gb300.adjoint import evidence_and_grad
    M, N, log_sigma = 512, 300, 0.3
    over = np.arange(5, M, 128)
    ds = _dead_set(M, P, N, over)
    out = evidence_and_grad(ds, math.log(1e19), log_sigma, tensor_cores=tensor_cores).cpu().numpy()
    keep = np.setdiff1d(np.arange(M), over)
    lw, y = ds.log_w.cpu().numpy()[keep], ds.y.cpu().numpy().astype(np.float64)
    s2 = math.exp(2.0 * log_sigma)
    ref = (np.log(np.exp(lw - lw.max()).sum()) + lw.max()
           - 0.5 * N * (math.log(2.0 * math.pi) + 2.0 * log_sigma) - 0.5 * (y @ y) / s2)
    # w = 0 in the other points: y^2 in fp32 chains of 32, N products
    assert abs(out[0] - ref) <= 40 * 2.0 ** -24 * 0.5 * (y @ y) / s2
    assert np.isnan(out[1]) and np.isnan(out[2])


@pytest.mark.parametrize("tensor_cores", [True, False])
def test_a_whole_range_of_overflowing_points(gpu_lib, tensor_cores):
    """The first 128 points all overflow: one block of the reduction has nothing finite, and the result
    is the one of the single block that takes all points."""
    from jaxns_gb300.adjoint import evidence_and_grad
    ds = _dead_set(512, 3, 300, np.arange(128))
    out = evidence_and_grad(ds, math.log(1e19), 0.3, tensor_cores=tensor_cores).cpu().numpy()
    assert np.isfinite(out[0]) and np.isnan(out[1]) and np.isnan(out[2])
