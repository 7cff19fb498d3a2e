"""The speculative sampler of small batches: every lane count the launcher takes, and the
thread-per-chain kernel above its last line, give the fp32 oracle's chains bit for bit."""
import numpy as np
import pytest

from conftest import assert_shell_exact, corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _spec(oracle_mod, D, S, K, prior, midpoint, n=42):
    from jaxns_gb300.engine import RunSpec, mvn_offset, mvn_params, shells_offset, shells_params
    kind, a, b = np.zeros(D, np.int32), np.full(D, -6.0), np.full(D, 12.0)
    if prior == "shells":
        c = np.zeros(D)
        c[0] = 3.5
        family, params, offset = 1, shells_params(c, -c, 2.0, 0.1), shells_offset(0.1)
    else:
        mu, cov = corr_gauss(D, D)
        family, params, offset = 0, mvn_params(mu, cov), mvn_offset(cov)
        if prior == "normal":
            kind, a, b = np.ones(D, np.int32), mu + 4.0, np.full(D, 1.5)  # posterior in the quantile's tail
        elif prior == "mixed":
            kind, a, b = (np.arange(D) % 2).astype(np.int32), np.where(np.arange(D) % 2, mu, -6.0), \
                np.where(np.arange(D) % 2, 2.0, 12.0)
    return RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=S, family=family, params=params,
                   prior_kind=kind, prior_a=a, prior_b=b, max_samples=40 * n, term_cond={"max_samples": 40 * n},
                   key=oracle_mod.PRNGKey(D + 100 * S), num_phantom=K, midpoint_shrink=midpoint, log_L_offset=offset)


# runs of 21 chains (one 64-chain item each): 32, 8 and 4 lanes per chain, then one thread per chain
@pytest.mark.parametrize("runs", [1, 20, 100, 400])
@pytest.mark.parametrize("D,S,K,prior,midpoint", [
    (1, 1, 0, "uniform", True), (2, 33, 0, "uniform", True), (7, 8, 2, "normal", True), (8, 40, 0, "normal", False),
    (9, 31, 0, "mixed", True), (16, 17, 3, "uniform", True), (10, 50, 0, "shells", True), (24, 9, 0, "shells", True),
    (48, 5, 1, "shells", False)])
def test_every_lane_count_matches_the_oracle(gpu_lib, oracle_mod, runs, D, S, K, prior, midpoint):
    from jaxns_gb300.engine import NSBatch
    spec = _spec(oracle_mod, D, S, K, prior, midpoint)
    b = NSBatch([spec] * runs, device="cuda")
    b.init()
    b.iterate(14)  # contours tight enough that slices outlast the uniforms prepared for them
    assert int(b.state()[0]["iterations"]) == 14
    live = b.live_view(0)["log_L_raw"].cpu().numpy()
    for at in (spec.shell_size - 1, spec.num_live_points - 2):  # the sampler's contour; a tight one (many shrinks)
        key = oracle_mod.PRNGKey(7 + at)
        b.slice_shell(torch.full((runs,), float(live[at])), torch.tensor(key.view(np.int32)).repeat(runs, 1))
        torch.cuda.synchronize()
        for r in {0, runs - 1}:
            assert_shell_exact(oracle_mod, b, r, live[at], key)


def test_evaluation_budget(gpu_lib, oracle_mod):
    """A slice that spends its evaluation budget takes its last point and reports it, on this
    kernel as on the thread-per-chain one."""
    from jaxns_gb300.engine import NSBatch
    spec = _spec(oracle_mod, 6, 12, 0, "uniform", True)
    out = []
    for runs in (1, 20, 100, 400):
        b = NSBatch([spec] * runs, device="cuda", max_evals_per_slice=3)
        b.init()
        top = float(b.live_view(0)["log_L_raw"][-2].item())
        key = torch.tensor(oracle_mod.PRNGKey(5).view(np.int32)).repeat(runs, 1)
        b.slice_shell(torch.full((runs,), top), key)
        torch.cuda.synchronize()
        s = spec.shell_size
        out.append((b.new_E[:s].cpu().numpy(), b.new_U_view(0).cpu().numpy(), b.new_L[:s].cpu().numpy()))
        assert int(b.state()[0]["status"]) == 2
    for o in out[1:]:
        for x, y in zip(o, out[0]):
            np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


# 201 chains per run (one item each): 16 / 8 / 4 proposals per round, then the warp-cooperative kernel
@pytest.mark.parametrize("runs", [1, 4, 16, 110])
@pytest.mark.parametrize("D,S,K,prior,midpoint", [
    (17, 1, 0, "uniform", True), (24, 21, 3, "uniform", False), (31, 33, 0, "mixed", True), (32, 16, 0, "normal", True),
    (33, 9, 2, "uniform", True), (50, 18, 0, "mixed", True), (64, 17, 0, "uniform", True)])
def test_wide_gaussians_match_the_oracle(gpu_lib, oracle_mod, runs, D, S, K, prior, midpoint):
    from jaxns_gb300.engine import NSBatch
    spec = _spec(oracle_mod, D, S, K, prior, midpoint, n=402)
    b = NSBatch([spec] * runs, device="cuda")
    b.init()
    b.iterate(14)  # contours tight enough that slices outlast the uniforms prepared for them
    assert int(b.state()[0]["iterations"]) == 14
    live = b.live_view(0)["log_L_raw"].cpu().numpy()
    for at in (spec.shell_size - 1, spec.num_live_points - 2):
        key = oracle_mod.PRNGKey(7 + at)
        b.slice_shell(torch.full((runs,), float(live[at])), torch.tensor(key.view(np.int32)).repeat(runs, 1))
        torch.cuda.synchronize()
        for r in {0, runs - 1}:
            assert_shell_exact(oracle_mod, b, r, live[at], key)
