"""Model.forward at the edges of its tiles, bit for bit the fp32 oracle; the linear-Gaussian points
(forward and initial live points) against the sum over rows in row order."""
import numpy as np
import pytest

from conftest import corr_gauss, model32_of_spec

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 127, 129, 256, 40000, 77901])  # one and two points per thread
@pytest.mark.parametrize("D,family,normal", [(1, 0, False), (9, 0, True), (10, 1, False), (64, 0, False)])
def test_forward_tiles(gpu_lib, oracle_mod, B, D, family, normal):
    from jaxns_gb300.engine import NSBatch, RunSpec, mvn_offset, mvn_params, shells_offset, shells_params
    c = np.zeros(D)
    c[0] = 3.5
    mu, cov = corr_gauss(D, D)
    params, off = (shells_params(c, -c, 2.0, 0.1), shells_offset(0.1)) if family else (mvn_params(mu, cov), mvn_offset(cov))
    spec = RunSpec(D=D, num_live_points=64, shell_size=32, num_slices=2, family=family, params=params,
                   prior_kind=np.full(D, int(normal), np.int32), prior_a=np.full(D, -6.0), prior_b=np.full(D, 12.0),
                   max_samples=640, term_cond={"dlogZ": 1e-4}, key=oracle_mod.PRNGKey(1), log_L_offset=off)
    b = NSBatch([spec])
    U = np.random.default_rng(B + D).random((B, D)).astype(np.float32)
    U[0, 0] = 0.0  # with a Normal prior: an infinite coordinate
    got = b.forward(0, torch.from_numpy(U)).cpu().numpy()
    m32 = model32_of_spec(oracle_mod, spec)
    m32.variant = 0  # Model.forward sums sequentially
    rows = np.unique(np.concatenate([np.arange(min(B, 300)), np.arange(max(0, B - 300), B)]))
    ref = oracle_mod.forward32(m32, U[rows]).astype(np.float64) + spec.log_L_offset
    np.testing.assert_array_equal(got[rows].view(np.uint32), ref.astype(np.float32).view(np.uint32))


@pytest.mark.parametrize("N,P,n", [(1, 1, 8), (127, 3, 9), (128, 64, 7), (129, 33, 8), (700, 12, 301)])
def test_linear_gaussian_points(gpu_lib, N, P, n):
    import jaxns_gb300 as gb
    from jaxns_gb300.engine import NSBatch
    g = np.random.default_rng(N * P)
    Phi, y = g.standard_normal((N, P)).astype(np.float32), g.standard_normal(N).astype(np.float32)

    def prior_model():
        w = yield gb.Prior(gb.Uniform(-np.ones(P), np.ones(P)), name="w")
        return w

    ns = gb.NestedSampler(gb.Model(prior_model, gb.LinearGaussianLikelihood(Phi, y, 0.5)), num_live_points=n, num_slices=2)
    other = ns.nested_sampler.run_spec(gb.random.PRNGKey(5), ns.normalise_term_cond(None))
    spec = ns.nested_sampler.run_spec(gb.random.PRNGKey(4), ns.normalise_term_cond(None))
    b = NSBatch([other, spec])  # the second run's points start inside a block of eight
    b.init()
    live = b.live_view(1)
    U, L = live["U"], live["log_L_raw"].cpu().numpy()
    np.testing.assert_array_equal(np.sort(L), L)
    fwd = b.forward(1, U).cpu().numpy()
    np.testing.assert_array_equal(fwd, (L.astype(np.float64) + spec.log_L_offset).astype(np.float32))
    w = -1.0 + 2.0 * U.cpu().numpy()
    r = y.astype(np.float64) - w @ Phi.astype(np.float64).T
    ref = -0.5 * (r * r).sum(1) / 0.25
    # N fp32 additions and N P products: relative error below (N + 2 P) 2^-24 of the sum
    np.testing.assert_allclose(L, ref, rtol=(N + 2 * P + 8) * 2.0 ** -24)
