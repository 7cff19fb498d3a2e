"""gbns_batch_init over runs of different families in one batch, which a caller of the C ABI can build,
with and without work items for the sampler."""
import ctypes

import numpy as np
import pytest

from conftest import corr_gauss

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", [True, False])
@pytest.mark.parametrize("lg_run", [0, 1, 2])
def test_every_run_gets_its_points(gpu_lib, oracle_mod, lg_run, items):
    """Three correlated Gaussians of D = 4, one of them turned into a linear-Gaussian run of 4 rows (as
    many parameters: Phi, y, sigma in place of mu, Linv, c0): the other runs' live sets stay those of the
    unchanged batch, and its own is that of the same run alone."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import NSBatch, RunSpec, mvn_offset, mvn_params
    D, n = 4, 40
    mu, cov = corr_gauss(D, 1)
    specs = [RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=2, family=0, params=mvn_params(mu, cov),
                     prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -10.0), prior_b=np.full(D, 20.0),
                     max_samples=4 * n, term_cond={"dlogZ": 1e-3}, key=oracle_mod.PRNGKey(7 + r), store_U=False,
                     log_L_offset=float(mvn_offset(cov))) for r in range(3)]
    ref = NSBatch(specs)
    ref.init()
    params = np.concatenate([np.eye(D).ravel(), np.zeros(D), [1.0]]).astype(np.float32)
    alone = NSBatch([RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=2, family=2, params=params, N=D,
                             prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -10.0), prior_b=np.full(D, 20.0),
                             max_samples=4 * n, term_cond={"dlogZ": 1e-3}, key=oracle_mod.PRNGKey(7 + lg_run),
                             store_U=False, log_L_offset=0.0)], lg_fused=False)
    alone.init()
    b = NSBatch(specs)
    words = torch.zeros(2, 4 * n * D, device="cuda")  # room for the FP64 points
    for p in range(2):
        b._b.live_U[p] = words[p].data_ptr()
    d = b._descs_host[lg_run]
    d.family, d.N, d.ucols = 2, D, 2 * D
    for r in range(3):
        b._descs_host[r].liveU_off = n * D * (r + (r > lg_run))
    b.t_runs.copy_(torch.frombuffer(bytearray(bytes(b._descs_host)), dtype=torch.uint8))
    b.fparams[lg_run * len(params):(lg_run + 1) * len(params)] = torch.from_numpy(params).cuda()
    if not items:
        for k in range(8):
            b._b.bucket_begin[k] = b._b.bucket_end[k] = 0
    _ffi.call("gbns_batch_init", ctypes.byref(b._b), b._stream())
    for r in range(3):
        got = b.live_L[0][r * n:(r + 1) * n].cpu().numpy()
        want = (alone.live_L[0] if r == lg_run else ref.live_L[0][r * n:(r + 1) * n]).cpu().numpy()
        np.testing.assert_array_equal(got, want)


def test_no_data_rows(gpu_lib, oracle_mod):
    """A linear-Gaussian run without data rows, which the C ABI does not refuse: log L is 0 at every
    point."""
    from jaxns_gb300 import _ffi
    from jaxns_gb300.engine import NSBatch, RunSpec
    D, n = 3, 16
    spec = RunSpec(D=D, num_live_points=n, shell_size=n // 2, num_slices=2, family=2,
                   params=np.full(D + 2, 0.5, np.float32), N=1, prior_kind=np.zeros(D, np.int32), prior_a=np.full(D, -1.0),
                   prior_b=np.full(D, 2.0), max_samples=4 * n, term_cond={"dlogZ": 1e-3}, key=oracle_mod.PRNGKey(7),
                   store_U=False, log_L_offset=0.0)
    b = NSBatch([spec], lg_fused=False)
    b.init()
    b._descs_host[0].N = 0
    b.t_runs.copy_(torch.frombuffer(bytearray(bytes(b._descs_host)), dtype=torch.uint8))
    U = torch.rand(20, D, dtype=torch.float64, device="cuda")
    np.testing.assert_array_equal(b.forward(0, U).cpu().numpy(), 0.0)
    _ffi.call("gbns_batch_init", ctypes.byref(b._b), b._stream())
    np.testing.assert_array_equal(b.live_L[0].cpu().numpy(), 0.0)
