"""Results of short runs: blocks that work alone, the same runs beside a long one (blocks that meet at
barriers), and one block per run in a large batch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _batch(ns, K):
    import jaxns_gb300 as gb
    from jaxns_gb300.engine import NSBatch, RunSpec, shells_offset, shells_params
    D = 3
    c = np.zeros(D)
    c[0] = 3.5
    specs = [RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=4, family=1, params=shells_params(c, -c, 2.0, 0.1),
                     prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -6.0), prior_b=np.full(D, 12.0),
                     max_samples=n * 40 * (1 + K), term_cond={"dlogZ": 1e-4}, num_phantom=K, key=gb.random.PRNGKey(n + r % 3),
                     store_U=True, log_L_offset=shells_offset(0.1)) for r, n in enumerate(ns)]
    b = NSBatch(specs)
    b.run(block=8)
    return b, b.results(with_U=True)


@pytest.mark.parametrize("n,K", [(2, 0), (30, 0), (60, 0), (20, 3), (26, 3)])
def test_short_runs(gpu_lib, n, K):
    ref_b, ref = _batch([n] * 100, K)
    longest = int(ref_b.state()["num_samples"].max())
    assert longest < 1600
    for ns in ([n], [n] * 3, [n] * 70, [n] * 3 + [400]):
        b, out = _batch(ns, K)
        for r in range(min(3, len(ns))):
            v, w = b.run_slices(r, out), ref_b.run_slices(r, ref)
            for f in ("samples_indices", "num_live_points", "log_L_samples", "nevals_sorted", "U_sorted"):
                np.testing.assert_array_equal(v[f].cpu().numpy(), w[f].cpu().numpy(), err_msg=f)
            # sums of the same fp32-pair terms in another grouping: a few units of 2^-48 per sample
            for f in ("log_X_mean", "log_dp_mean", "scalars"):
                np.testing.assert_allclose(v[f].cpu().numpy(), w[f].cpu().numpy(), rtol=1e-11, atol=1e-11, err_msg=f)
