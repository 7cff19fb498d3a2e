"""The warp-cooperative sampler above the speculative kernel's last line: flattened normals with
queued tails, per-lane norms and bounds, bit for bit the fp32 oracle's chains."""
import numpy as np
import pytest

from conftest import assert_shell_exact, corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,runs,normal", [(17, 60, False), (31, 60, True), (32, 56, False), (33, 34, False), (47, 30, True),
                                           (63, 30, False), (64, 30, True)])
def test_warp_directions(gpu_lib, oracle_mod, D, runs, normal):
    from jaxns_gb300.engine import NSBatch, RunSpec, mvn_offset, mvn_params
    n = 1000
    mu, cov = corr_gauss(D, D)
    kind, a, b = (np.ones(D, np.int32), mu + 1.0, np.full(D, 1.5)) if normal else (np.zeros(D, np.int32), np.full(D, -6.0),
                                                                                     np.full(D, 12.0))
    spec = RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=3, family=0, params=mvn_params(mu, cov), prior_kind=kind,
                   prior_a=a, prior_b=b, max_samples=40 * n, term_cond={"max_samples": 40 * n}, key=oracle_mod.PRNGKey(D),
                   log_L_offset=mvn_offset(cov))
    b = NSBatch([spec] * runs, device="cuda")
    b.init()
    b.iterate(3)
    live = b.live_view(0)["log_L_raw"].cpu().numpy()
    key = oracle_mod.PRNGKey(11)
    b.slice_shell(torch.full((runs,), float(live[n // 2])), torch.tensor(key.view(np.int32)).repeat(runs, 1))
    torch.cuda.synchronize()
    for r in (0, runs - 1):
        assert_shell_exact(oracle_mod, b, r, live[n // 2], key)
